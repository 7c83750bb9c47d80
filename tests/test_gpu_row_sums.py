"""Vertex weights and modularity at the edges of their row groups: rows of 0 to
thousands of entries around 8, 32, 128 and 512, absent vertices, with unit,
whole and fractional weights, against numpy's sums.

Weights are multiples of 1/2, so every sum of them is exact in any order;
modularity also divides and adds squares (relative rounding 2^-53 for each of
at most 2^13 additions).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1024, 4097]


@pytest.mark.parametrize("weights", ["unit", "whole", "half"])
def test_rows_of_every_group(cuda, lvg, weights):
    rng = np.random.default_rng(5)
    k, leaf = len(DEGREES), 200  # rows 1..k to leaves from id 200 on; ids between are absent
    src = np.concatenate([np.full(d, 1 + i) for i, d in enumerate(DEGREES)])
    dst = np.concatenate([leaf + rng.choice(4200, d, replace=False) for d in DEGREES])
    w = rng.integers(1, 9, len(src)).astype(np.float32)
    w = {"unit": np.ones_like(w), "whole": w, "half": w * np.float32(0.5)}[weights]
    x = lvg.csr_from_edges(leaf + 4300, np.concatenate([src, dst]).astype(np.uint32),
                           np.concatenate([dst, src]).astype(np.uint32), np.concatenate([w, w]))
    x.exists[k + 1:leaf] = 0
    deg = np.diff(x.offsets).astype(np.int64)
    assert set(DEGREES) <= set(deg[1:k + 1]) and not deg[k + 1:leaf].any()
    row, total = np.repeat(np.arange(x.span), deg), x.weights.astype(np.float64)
    X = cuda.Graph(x)
    own = np.bincount(row, weights=total, minlength=x.span)
    assert np.array_equal(cuda.louvain_static(X).vertexWeight, own)
    assert np.array_equal(X.vertex_weights(), own)

    memb = rng.integers(0, 40, x.span).astype(np.uint32)
    memb[leaf:] = np.where(rng.random(x.span - leaf) < 0.5, 7, memb[leaf:])  # one large community
    M = total.sum() / 2
    inside = total[memb[row] == memb[x.keys]].sum()
    tot = np.bincount(memb, weights=own)
    want = inside / (2 * M) - (tot * tot).sum() / (4 * M * M)
    assert X.modularity(memb) == pytest.approx(want, abs=2.0 ** -40)

    for u in (leaf + 5, k + 5):  # an id that is no vertex: refused, for an absent vertex too
        bad = memb.copy()
        bad[u] = x.span
        with pytest.raises(lvg.LvgError):
            X.modularity(bad)
    assert X.modularity(memb) == pytest.approx(want, abs=2.0 ** -40)
