"""Vertex weights and modularity over the range of spans: a vertex per warp or
four (up to 9728 vertices on 152 SMs, and more), 8 to 256 vertices per block, long
rows among short ones, against numpy's sums. Weights are multiples of 1/2: every
sum is exact in any order; modularity also divides and adds squares (relative
rounding 2^-53 for each of at most 2^20 additions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONG = [128, 129, 511, 513, 2047, 2048, 2049, 4097, 6500]


@pytest.mark.parametrize("weights", ["unit", "half"])
@pytest.mark.parametrize("span", [7000, 9728, 9729, 20001, 38913, 160000, 330003])
def test_spans(cuda, lvg, span, weights):
    rng = np.random.default_rng(span)
    u = np.arange(1, span)
    rows = rng.choice(u, 4 * len(LONG), replace=False)  # four of each long degree, anywhere
    src = np.concatenate([np.full(d, x) for x, d in zip(rows, np.repeat(LONG, 4))] + [u])
    dst = np.concatenate([rng.choice(u, d, replace=False) for d in np.repeat(LONG, 4)] + [1 + u % (span - 1)])
    a, b = np.minimum(src, dst).astype(np.uint64), np.maximum(src, dst).astype(np.uint64)
    pair = np.unique((a << np.uint64(32) | b)[a != b])
    a, b = (pair >> np.uint64(32)).astype(np.uint32), (pair & np.uint64(0xffffffff)).astype(np.uint32)
    w = rng.integers(1, 9, len(a)).astype(np.float32) * np.float32(0.5)
    if weights == "unit":
        w[:] = 1
    x = lvg.csr_from_edges(span - 1, np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w]))
    assert x.span == span and (np.diff(x.offsets) > 2048).any()
    row, total = np.repeat(np.arange(span), np.diff(x.offsets).astype(np.int64)), x.weights.astype(np.float64)
    own = np.bincount(row, weights=total, minlength=span)
    X = cuda.Graph(x)
    assert np.array_equal(X.vertex_weights(), own)
    assert np.array_equal(cuda.louvain_static(X).vertexWeight, own)
    memb = rng.integers(0, 40, span).astype(np.uint32)
    memb[span // 2:] = 7
    M = total.sum() / 2
    tot = np.bincount(memb, weights=own)
    want = total[memb[row] == memb[x.keys]].sum() / (2 * M) - (tot * tot).sum() / (4 * M * M)
    assert X.modularity(memb) == pytest.approx(want, abs=2.0 ** -32)
