"""Phases whose blocks list more vertices of a class than shared memory holds
(1920 a block, at most one block per SM): lists and moves in device memory,
against the launch-by-launch path, bit for bit (unit weights)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LISTED = 1920 * 152


@pytest.mark.parametrize("n,colors", [(LISTED - 4000, 1), (LISTED + 4000, 1), (600000, 1), (650000, 2)])
def test_lists_in_device_memory(cuda, lvg, n, colors):
    x = lvg.planted_partition(n, 300, 12, 0.8, 5)
    vt = np.diff(x.offsets).astype(np.float64)
    prior = np.arange(x.span, dtype=np.uint32), vt, vt
    o = cuda.LouvainOptions(deterministic=True, colors=colors, maxPasses=2)
    out = []
    for graphs in (0, 1):
        g = cuda.Graph(x)
        cuda.set_tuning(g, level_graphs=graphs)
        out.append([cuda.louvain_static(g, o), cuda.louvain_naive_dynamic(g, cuda.HostBatch.empty(), *prior, o)])
        assert (g.stats()["level_graphs"] > 0) == bool(graphs)
    for a, b in zip(*out):
        assert (a.iterations, a.passes, a.affectedVertices) == (b.iterations, b.passes, b.affectedVertices)
        for f in ("membership", "vertexWeight", "communityWeight"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f


def test_lists_in_device_memory_fractional(cuda, lvg):
    """The same with weights of 1/2 to 4 (sums exact in any order)."""
    x = lvg.planted_partition(600000, 300, 12, 0.8, 5)
    u = np.repeat(np.arange(x.span), np.diff(x.offsets).astype(np.int64))
    x.weights[:] = 0.5 * (1 + (np.minimum(u, x.keys) * 7919 + np.maximum(u, x.keys) * 104729) % 8)
    o = cuda.LouvainOptions(deterministic=True, colors=1, maxPasses=2)
    out = []
    for graphs in (0, 1):
        g = cuda.Graph(x)
        cuda.set_tuning(g, level_graphs=graphs)
        out.append(cuda.louvain_static(g, o))
    a, b = out
    assert (a.iterations, a.passes) == (b.iterations, b.passes)
    assert np.array_equal(a.membership, b.membership) and np.array_equal(a.communityWeight, b.communityWeight)
