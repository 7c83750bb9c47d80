"""Dynamic runs on levels of large vertices, on both sides of the rule that sends
them launch by launch: the deterministic result is the same on either path, bit
for bit, the asynchronous one of the same quality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# vertices, community, degree, weights; launch by launch when asynchronous, when deterministic
@pytest.mark.parametrize("n,block,degree,weights,launches", [
    (2000, 1000, 300, "unit", (False, False)),
    (30000, 1000, 300, "unit", (True, False)),    # 9M edges at degree 257-512
    (30000, 1000, 300, "half", (True, False)),
    (9000, 4500, 3200, "unit", (True, True)),     # 20M edges above degree 2048
    (9000, 4500, 3200, "half", (True, True)),
])
def test_route_and_result(cuda, lvg, n, block, degree, weights, launches):
    x = lvg.planted_partition(n, block, degree, 0.9, 7)
    if weights == "half":
        u = np.repeat(np.arange(x.span), np.diff(x.offsets).astype(np.int64))
        x.weights[:] = 0.5 * (1 + (np.minimum(u, x.keys) * 7919 + np.maximum(u, x.keys) * 104729) % 4)
    r = cuda.louvain_static(cuda.Graph(x), cuda.LouvainOptions(deterministic=True))
    q = np.array(r.membership)
    q[1::7] = np.arange(x.span)[1::7]  # some vertices on their own again
    vt = np.array(r.vertexWeight)
    prior = q, vt, np.bincount(q, weights=vt, minlength=x.span)
    none = cuda.HostBatch.empty()
    for deterministic in (False, True):
        o = cuda.LouvainOptions(deterministic=deterministic, maxPasses=1)
        out = []
        for graphs in (1, 0):
            g = cuda.Graph(x)
            cuda.set_tuning(g, level_graphs=graphs)
            out.append(cuda.louvain_naive_dynamic(g, none, *prior, o))
            if graphs:
                assert (g.stats()["kernel_launches"] > 40) == launches[deterministic]
                # a frontier run of a small batch looks at few vertices
                b = lvg.random_batch(x, 4, 0.8, seed=5)
                cuda.louvain_dynamic_frontier(g, b, *prior, o)
                assert g.stats()["kernel_launches"] <= 40
        a, b = out
        if deterministic:
            assert a.iterations == b.iterations
            for f in ("membership", "vertexWeight", "communityWeight"):
                assert np.array_equal(getattr(a, f), getattr(b, f)), f
        else:
            assert g.modularity(a.membership) == pytest.approx(g.modularity(b.membership), abs=0.005)


@pytest.mark.parametrize("weights,launches", [("unit", False), ("half", True)])
def test_static_route_and_result(cuda, lvg, weights, launches):
    """A deterministic static run on vertices above degree 2048 goes launch by
    launch when its weights are fractional."""
    x = lvg.planted_partition(9000, 4500, 3200, 0.9, 7)
    if weights == "half":
        u = np.repeat(np.arange(x.span), np.diff(x.offsets).astype(np.int64))
        x.weights[:] = 0.5 * (1 + (np.minimum(u, x.keys) * 7919 + np.maximum(u, x.keys) * 104729) % 4)
    out = []
    for graphs in (1, 0):
        g = cuda.Graph(x)
        cuda.set_tuning(g, level_graphs=graphs)
        out.append(cuda.louvain_static(g, cuda.LouvainOptions(deterministic=True, maxPasses=1)))
        if graphs:
            assert (g.stats()["kernel_launches"] > 40) == launches
    a, b = out
    assert a.iterations == b.iterations
    for f in ("membership", "vertexWeight", "communityWeight"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
