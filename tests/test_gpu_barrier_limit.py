"""A phase whose barrier wait is given up (lvg_set_barrier_polls: here after one
poll) ends with LVG_ETIMEOUT and leaves nothing behind: the next runs on the same
graph and states equal those of fresh ones, bit for bit. The graph has hubs,
whose partial sums, counts and resident tables live from one phase to the next."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def base(cuda):
    # R-MAT scale 16, edge factor 48: ~40 vertices above degree 8192, unit weights
    x = cuda.rmat(16, 48, seed=77)
    r = cuda.louvain_static(cuda.Graph(x), cuda.LouvainOptions(deterministic=True))
    return x, (r.membership, r.vertexWeight, r.communityWeight)


def _times_out(cuda, G, call):
    G.set_barrier_polls(1)
    with pytest.raises(cuda.LvgError) as e:
        call()
    assert e.value.code == cuda.LVG_ETIMEOUT and "barrier" in str(e.value)
    G.set_barrier_polls(0)


def _same(a, b):
    assert (a.iterations, a.passes, a.affectedVertices) == (b.iterations, b.passes, b.affectedVertices)
    for f in ("membership", "vertexWeight", "communityWeight"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("colors", [1, 16])
def test_next_runs_equal_a_fresh_graph(cuda, base, colors):
    x, prior = base
    o = cuda.LouvainOptions(deterministic=True, colors=colors)
    none = cuda.HostBatch.empty()
    F = cuda.Graph(x)
    # (a hub's neighbours lie in eight communities alike, its own among them: its
    # own one's sum, half made when the phase ends, decides whether it moves)
    q = (1 + np.arange(x.span) % 8).astype(np.uint32)
    prior = q, prior[1], np.bincount(q, weights=prior[1], minlength=x.span)
    fresh = [cuda.louvain_naive_dynamic(F, none, *prior, o), cuda.louvain_static(F, o)]
    G = cuda.Graph(x)
    for _ in range(3):
        _times_out(cuda, G, lambda: cuda.louvain_naive_dynamic(G, none, *prior, o))
        _same(cuda.louvain_naive_dynamic(G, none, *prior, o), fresh[0])
        _times_out(cuda, G, lambda: cuda.louvain_static(G, o))
        _same(cuda.louvain_static(G, o), fresh[1])


def test_union_after_a_timeout(cuda, base):
    x, _ = base
    o = cuda.LouvainOptions(deterministic=True)
    U = cuda.Graph.union([cuda.Graph(x), cuda.Graph(cuda.planted_partition(20000, 100, 16, 0.8, 3))])
    fresh = cuda.louvain_static_union(U, o)
    fresh = [(np.array(r.membership), np.array(r.communityWeight)) for r in fresh]
    _times_out(cuda, U, lambda: cuda.louvain_static_union(U, o))
    for r, (m, ct) in zip(cuda.louvain_static_union(U, o), fresh):
        assert np.array_equal(r.membership, m) and np.array_equal(r.communityWeight, ct)


def test_resident_tables_after_a_timeout(cuda, base):
    """A frontier run in place: its state's tables were half brought up to date."""
    x, prior = base
    o = cuda.LouvainOptions(deterministic=True)
    G = cuda.Graph(x)
    db = cuda.DeviceBatch(G, cuda.random_batch(x, 3000, seed=5))
    G.apply_batch(db)
    st = cuda.State(G)
    st.set(*prior)
    cuda.run_resident(G, cuda.METHOD_FRONTIER, db, st, st, o)  # (with tables)
    assert G.stats()["hub_tables_built"] == 1
    more = cuda.DeviceBatch(G, cuda.random_batch(x, 4000, seed=6))
    G.apply_batch(more)
    _times_out(cuda, G, lambda: cuda.run_resident(G, cuda.METHOD_FRONTIER, more, st, st, o))
    left = st.get()  # whatever the run left is a state: go on from it here and in a fresh graph
    assert left[0].max() < G.span
    batch = cuda.DeviceBatch(G, cuda.random_batch(x, 3000, seed=7))
    G.apply_batch(batch)
    cuda.run_resident(G, cuda.METHOD_FRONTIER, batch, st, st, o)
    assert G.stats()["hub_tables_built"] == 1
    F = cuda.Graph(G.download())
    fs = cuda.State(F)
    fs.set(*left)
    cuda.run_resident(F, cuda.METHOD_FRONTIER, cuda.DeviceBatch(F, batch.download()), fs, fs, o)
    for a, b in zip(st.get(), fs.get()):
        assert np.array_equal(a, b)
