"""Deterministic mode with weights whose FP32 sums depend on their order: a
vertex of degree up to 512 is decided from one order of its row, so repeated
runs agree bit for bit, and so do the phase kernel and the launch-by-launch
path. The vertices here have the same weights to two communities in another
order each, so which one they join is a matter of rounding alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tied(lvg, half, own, seed):
    """300 vertices with `half` neighbours of the same weights in each of two
    communities of 600, and `own` neighbours in their own. Weights are multiples
    of 2^-24: the communities' FP64 totals are exact in any order, so only the
    rows' FP32 sums are not."""
    rng = np.random.default_rng(seed)

    def weights(n):
        return rng.integers(1, 1 << 24, n).astype(np.float32) * np.float32(2.0 ** -24)

    base = weights(half)
    blocks = [1 + np.arange(600), 601 + np.arange(600)]
    u = 1201 + np.arange(300)
    src, dst, w = [], [], []
    for x in u:
        for b in blocks:
            src.append(np.full(half, x))
            dst.append(rng.choice(b, half, replace=False))
            w.append(rng.permutation(base))
        mine = 1501 + (x - 1201) * own + np.arange(own)
        src.append(np.full(own, x))
        dst.append(mine)
        w.append(weights(own) * np.float32(0.125))
    s, t, w = (np.concatenate(a) for a in (src, dst, w))
    n = 1500 + 300 * own
    g = lvg.csr_from_edges(n, np.concatenate([s, t]).astype(np.uint32), np.concatenate([t, s]).astype(np.uint32),
                           np.concatenate([w, w]))
    assert (np.diff(g.offsets)[u] == 2 * half + own).all()
    q = np.arange(g.span, dtype=np.uint32)
    q[blocks[0]], q[blocks[1]] = 1, 601
    q[1501:] = np.repeat(u, own)
    row = np.repeat(np.arange(g.span), np.diff(g.offsets).astype(np.int64))
    vt = np.bincount(row, weights=g.weights.astype(np.float64), minlength=g.span)
    return g, (q, vt, np.bincount(q, weights=vt, minlength=g.span)), u


# degrees of one, two and four times 32 lanes, both sides of each group's last degree
@pytest.mark.parametrize("half,own", [(15, 2), (15, 3), (30, 4), (31, 3), (62, 4), (63, 3), (125, 6), (126, 5), (250, 12)])
def test_order_of_a_row_is_fixed(cuda, lvg, half, own):
    g, prior, u = _tied(lvg, half, own, 2 * half + own)
    o = cuda.LouvainOptions(deterministic=True, colors=1, maxPasses=1, maxIterations=1)
    runs = []
    for graphs, repeats in ((1, 6), (0, 2)):
        G = cuda.Graph(g)
        cuda.set_tuning(G, level_graphs=graphs)
        for _ in range(repeats):
            r = cuda.louvain_naive_dynamic(G, cuda.HostBatch.empty(), *prior, o)
            runs.append((np.array(r.membership), np.array(r.communityWeight)))
        assert (G.stats()["level_graphs"] > 0) == bool(graphs)
    joined = runs[0][0][u]
    assert (joined == 1).any() and (joined == 601).any()  # rounding decided
    for m, ct in runs[1:]:
        assert np.array_equal(m, runs[0][0])
        assert np.array_equal(ct, runs[0][1])
