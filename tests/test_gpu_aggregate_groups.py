"""Aggregation at the edges of its groupings: communities whose total degree
lies at both sides of every bin's end and of a chunk, one of several hash
partitions (more than 8192 neighbour communities), members of degree 1 to
thousands, with unit, whole and fractional weights, against the sums numpy
takes per pair of communities.

Weights are multiples of 1/2 whose FP32 sums are exact in any order (below
2^23), so equality is the right tolerance.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 70000
# total degrees of the communities made of ring vertices (degree 4 each)
RINGS = [4, 8, 12, 32, 36, 64, 68, 128, 132, 256, 260, 512, 516, 2048, 2052, 4096, 4100, 8192, 8196, 12288, 16388]


@pytest.fixture(scope="module")
def case(lvg):
    """(sources, targets, membership): ids 1..N on a ring of degree 4, then vertices of long
    rows and leaves of degree 1, which with a stretch of the ring make one large community."""
    rng = np.random.default_rng(3)
    u = np.arange(1, N + 1)
    src, dst = [u, u], [u % N + 1, (u + 1) % N + 1]
    memb = np.arange(N + 8000 + 1)
    at = 1
    for t in RINGS:
        memb[at:at + t // 4] = at
        at += t // 4
    big = at  # the large community: 3000 ring vertices, four long rows, 7000 leaves of one of them
    memb[big:big + 3000] = big
    for i, d in enumerate([65, 700, 9000, 30000]):
        src.append(np.full(d, N + 1 + i))
        dst.append(rng.choice(u, d, replace=False))
        memb[N + 1 + i] = big
    leaves = np.arange(N + 5, N + 7005)
    src.append(leaves)
    dst.append(np.full(len(leaves), N + 1))
    memb[leaves] = big
    return np.concatenate(src), np.concatenate(dst), memb.astype(np.uint32)


@pytest.mark.parametrize("weights", ["unit", "whole", "half"])
def test_every_total_degree_group(cuda, lvg, case, weights):
    s, t, memb = case
    pair = np.unique(np.minimum(s, t).astype(np.uint64) << np.uint64(32) | np.maximum(s, t).astype(np.uint64))
    a, b = (pair >> np.uint64(32)).astype(np.uint32), (pair & np.uint64(0xffffffff)).astype(np.uint32)
    w = np.random.default_rng(9).integers(1, 9, len(a)).astype(np.float32)
    w = {"unit": np.ones_like(w), "whole": w, "half": w * np.float32(0.5)}[weights]
    x = lvg.csr_from_edges(len(memb) - 1, np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w]))
    assert x.span == len(memb)
    ren, cn, off, keys, sums = cuda.aggregate(cuda.Graph(x), memb)
    live = np.unique(memb[x.exists.astype(bool)])
    assert cn == len(live)
    ex = x.exists.astype(bool)
    assert np.array_equal(ren[ex], np.searchsorted(live, memb[ex]).astype(np.uint32))
    # numpy's sums per (community, neighbour community)
    row = np.repeat(np.arange(x.span), np.diff(x.offsets).astype(np.int64))
    pc = ren[row].astype(np.uint64) << np.uint64(32) | ren[x.keys].astype(np.uint64)
    want, inv = np.unique(pc, return_inverse=True)
    total = np.bincount(inv, weights=x.weights.astype(np.float64))
    got = np.repeat(np.arange(cn, dtype=np.uint64), np.diff(off).astype(np.int64)) << np.uint64(32) | keys.astype(np.uint64)
    order = np.argsort(got, kind="stable")
    assert np.array_equal(got[order], want)
    assert np.array_equal(sums[order], total)
    assert np.diff(off).max() > 16384  # a row of several partitions
