"""Deterministic phases whose blocks share their large vertices and the rows of
large movers (enough vertices of degree 513-8192 in a class), on both sides of
that rule and of the one for rows marked by a warp, against the launch-by-launch
path: memberships and totals bit for bit (weights are multiples of 1/2 whose
sums are exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same_as_launches(cuda, x, dynamic=False, **opts):
    """A static run, or a naive-dynamic one from singletons (totals of the caller's)."""
    out = []
    row = np.repeat(np.arange(x.span), np.diff(x.offsets).astype(np.int64))
    own = np.bincount(row, weights=x.weights.astype(np.float64), minlength=x.span)
    prior = np.arange(x.span, dtype=np.uint32), own, own
    for graphs in (0, 1):
        g = cuda.Graph(x)
        cuda.set_tuning(g, level_graphs=graphs)
        o = cuda.LouvainOptions(deterministic=True, **opts)
        out.append(cuda.louvain_naive_dynamic(g, cuda.HostBatch.empty(), *prior, o) if dynamic
                   else cuda.louvain_static(g, o))
        assert (g.stats()["level_graphs"] > 0) == bool(graphs)
    a, b = out
    assert (a.iterations, a.passes) == (b.iterations, b.passes) and a.iterations > 1
    for f in ("membership", "vertexWeight", "communityWeight"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("weights", ["unit", "whole", "half"])
@pytest.mark.parametrize("large", [500, 4000])
def test_large_vertices(cuda, lvg, large, weights):
    rng = np.random.default_rng(large)
    small = 60000
    degrees = np.concatenate([rng.integers(520, 900, large), [2048, 2500, 9000, 14000, 20000],
                              rng.integers(2300, 9000, 60)])
    src = np.repeat(small + 1 + np.arange(len(degrees)), degrees)
    group = np.repeat(rng.integers(0, 8, len(degrees)), degrees)  # most neighbours out of one of 8 ranges
    dst = 1 + np.where(rng.random(len(src)) < 0.7, group * 7500 + rng.integers(0, 7500, len(src)),
                       rng.integers(0, small, len(src)))
    pair = np.unique(dst.astype(np.uint64) << np.uint64(32) | src.astype(np.uint64))
    a, b = (pair >> np.uint64(32)).astype(np.uint32), (pair & np.uint64(0xffffffff)).astype(np.uint32)
    degree = np.bincount(b)  # (repeats taken out)
    assert ((degree > 512).sum() > 2500) == (large == 4000) and (degree > 2048).sum() > 30 and degree.max() > 8192
    w = rng.integers(1, 5, len(a)).astype(np.float32)
    w = {"unit": np.ones_like(w), "whole": w, "half": w * np.float32(0.5)}[weights]
    x = lvg.csr_from_edges(small + len(degrees), np.concatenate([a, b]), np.concatenate([b, a]),
                           np.concatenate([w, w]))
    _same_as_launches(cuda, x, colors=1, maxPasses=2)
    _same_as_launches(cuda, x, colors=3, maxPasses=2)
    _same_as_launches(cuda, x, dynamic=True, colors=1, maxPasses=2)


@pytest.mark.parametrize("dynamic", [False, True])
@pytest.mark.parametrize("n", [4000, 90000])
def test_rows_of_movers(cuda, lvg, n, dynamic):
    _same_as_launches(cuda, lvg.planted_partition(n, 300, 60, 0.8, 5), colors=1, dynamic=dynamic)
