"""lvg_graph_trim(1) leaves a graph with its rows, its workspace and little else,
whatever calls it has served: the serving loop admits graphs by the bytes they
hold after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_leave_no_scratch_behind(cuda, lvg):
    H, G = (cuda.Graph.rmat(18, 16, seed=5) for _ in range(2))  # hubs, communities above total degree 8192
    b = cuda.DeviceBatch.generate(G, 100, 400, seed=6).download()
    for g in (H, G):  # the workspace, grown by the same batch
        g.modularity(np.zeros(H.span, np.uint32))
        b = g.apply_batch(b)  # (tidied)
        undo = lvg.HostBatch(b.ins_src, b.ins_dst, b.ins_w, b.del_src, b.del_dst, b.del_w)
        g.apply_batch(undo)
    H.trim(1)
    det = cuda.LouvainOptions(deterministic=True)
    first = cuda.louvain_static(G, det)
    cuda.louvain_static(G, cuda.LouvainOptions())
    cuda.louvain_static(G, cuda.LouvainOptions(deterministic=True, colors=1))  # long lists of one class
    cuda.set_tuning(G, level_graphs=0)  # the launches' tables
    cuda.louvain_static(G, det)
    cuda.set_tuning(G, level_graphs=1)
    assert (np.diff(G.download().offsets) > 8192).any()
    G.apply_batch(b)
    prior = first.membership, first.vertexWeight, first.communityWeight
    for method in (cuda.louvain_naive_dynamic, cuda.louvain_dynamic_frontier):  # (the second builds hub tables)
        method(G, b, *prior, det)
    G.apply_batch(undo)
    G.trim(1)
    # the hubs' index map (4 bytes a vertex) and plans
    assert G.device_bytes() - H.device_bytes() <= 4 * G.span + (1 << 20)
    again = cuda.louvain_static(G, det)
    for f in ("membership", "vertexWeight", "communityWeight"):
        assert np.array_equal(getattr(again, f), getattr(first, f))


def test_union_runs_after_a_trim(cuda):
    U = cuda.Graph.union([cuda.Graph.planted_partition(n, 100, 12, 0.8, n) for n in (900, 5000, 20000)])
    o = cuda.LouvainOptions(deterministic=True)
    a = [np.array(r.membership) for r in cuda.louvain_static_union(U, o)]
    U.trim(1)
    assert all(np.array_equal(r.membership, m) for r, m in zip(cuda.louvain_static_union(U, o), a))
