"""A level's local-moving phase as one cooperative kernel: every degree at the
edge of the kernel's groupings (tiles of 4/8/16/32 lanes, 1/4/8/32 warps, hub
chunks and their hash partitions), with unit, whole and fractional weights (the
three ways its tables add), bit for bit against the oracle's replay of the
deterministic rule.

Weights are multiples of 1/2 whose FP32 sums are exact in any order (below
2^23), so equality is the right tolerance.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# both sides of every bin's last degree, of a hub chunk and of a partition
DEGREES = [1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 2047, 2048, 2049, 8191, 8192, 8193,
           12289, 16385, 30001]
N = 40000


@pytest.fixture(scope="module")
def edges():
    """A vertex of each degree above among N others in blocks of 50 (communities)."""
    rng = np.random.default_rng(11)
    src, dst = [], []
    u = np.arange(1, N + 1)
    for step in (1, 2, 3, 7):  # a ring lattice within each block
        v = (u - 1) // 50 * 50 + (u - 1 + step) % 50 + 1
        src.append(u)
        dst.append(v)
    for i, d in enumerate(DEGREES):
        src.append(np.full(d, N + 1 + i))
        dst.append(rng.choice(u, d, replace=False))
    s, t = np.concatenate(src), np.concatenate(dst)
    return s.astype(np.uint32), t.astype(np.uint32)


def _graph(lvg, edges, weights):
    s, t = edges
    a, b = np.minimum(s, t).astype(np.uint64), np.maximum(s, t).astype(np.uint64)
    pair = np.unique(a << np.uint64(32) | b)
    a, b = (pair >> np.uint64(32)).astype(np.uint32), (pair & np.uint64(0xffffffff)).astype(np.uint32)
    w = np.random.default_rng(5).integers(1, 9, len(a)).astype(np.float32)
    w = {"unit": np.ones_like(w), "whole": w, "half": w * np.float32(0.5)}[weights]
    g = lvg.csr_from_edges(N + len(DEGREES), np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w]))
    deg = np.diff(g.offsets).astype(np.int64)
    assert np.array_equal(deg[N + 1:], DEGREES)
    return g


@pytest.mark.parametrize("weights", ["unit", "whole", "half"])
@pytest.mark.parametrize("colors", [1, 5, 16])
def test_every_degree_group_matches_cpu_replay(cuda, orc, lvg, edges, weights, colors):
    x = _graph(lvg, edges, weights)
    o = cuda.LouvainOptions(deterministic=True, colors=colors, maxIterations=6, maxPasses=3)
    G = cuda.Graph(x)
    r = cuda.louvain_static(G, o)
    from oracle import oracle as O
    m, vt, ct, info = orc.louvain(x, 0, threads=8, sync=True, colors=colors,
                                  opts=O.options(maxIterations=6, maxPasses=3))
    assert np.array_equal(r.membership, m)
    assert np.array_equal(r.vertexWeight, vt)
    assert np.array_equal(r.communityWeight, ct)
    assert (r.iterations, r.passes, r.affectedVertices) == (info["iterations"], info["passes"],
                                                            info["affectedVertices"])
    st = G.stats()
    assert st["level_graphs"] >= r.passes  # the phases ran as one launch each
    # the launch-by-launch path: the same result and the same work
    H = cuda.Graph(x)
    cuda.set_tuning(H, level_graphs=0)
    s = cuda.louvain_static(H, o)
    assert np.array_equal(r.membership, s.membership) and np.array_equal(r.communityWeight, s.communityWeight)
    for k in ("move_vertices", "move_edges", "moves", "move_bin_vertices", "move_bin_edges"):
        assert st[k] == H.stats()[k], k


@pytest.mark.parametrize("scale", [1, 2])
def test_totals_around_2_31(cuda, lvg, scale):
    """Whole weights whose total lies below 2^31 (gains from integer totals) and
    above (FP64), with community totals beyond FP32's 2^24: the launch-by-launch
    path's FP64 totals, bit for bit. One pass: its FP32 sums per vertex and
    community stay below 2^24, exact in any order."""
    x = lvg.planted_partition(4096, 256, 256, 0.5, 3)
    u = np.repeat(np.arange(x.span), np.diff(x.offsets).astype(np.int64))
    x.weights[:] = scale * (1500 + (np.minimum(u, x.keys) * 7919 + np.maximum(u, x.keys) * 104729) % 1000)
    total = x.weights.astype(np.float64).sum()
    assert 2 ** 30 < total / scale < 2 ** 31 and (total >= 2 ** 31) == (scale == 2)
    out = []
    for graphs in (0, 1):
        g = cuda.Graph(x)
        cuda.set_tuning(g, level_graphs=graphs)
        r = cuda.louvain_static(g, cuda.LouvainOptions(deterministic=True, maxPasses=1))
        assert (g.stats()["level_graphs"] > 0) == bool(graphs)
        out.append(r)
    assert out[1].communityWeight.max() > 2 ** 24
    for f in ("membership", "vertexWeight", "communityWeight"):
        assert np.array_equal(getattr(out[0], f), getattr(out[1], f))
