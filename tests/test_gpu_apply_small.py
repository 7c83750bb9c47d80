"""Batches on both sides of the one-block plan (2048 entries a list), with
repeats, absent deletions, present insertions, sources in one list or both:
the updated graph and the tidied batch against
numpy's set operations (integers and copied weights, so equality)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(x):
    row = np.repeat(np.arange(x.span, dtype=np.uint64), np.diff(x.offsets).astype(np.int64))
    return row << np.uint64(32) | x.keys.astype(np.uint64)


@pytest.mark.parametrize("nd,ni", [(0, 1), (1, 0), (31, 33), (63, 64), (500, 2048), (2048, 0), (2048, 2048),
                                   (2049, 5), (0, 2049), (3000, 3000)])
def test_sizes(cuda, lvg, nd, ni):
    rng = np.random.default_rng(nd * 7 + ni)
    x = lvg.rmat(11, 6, seed=9)
    x.weights[:] = rng.integers(1, 50, len(x.weights)).astype(np.float32)
    old = _pairs(x)
    any_pair = lambda n: (rng.integers(1, x.span, n).astype(np.uint64) << np.uint64(32)
                          | rng.integers(1, x.span, n).astype(np.uint64))
    d = np.concatenate([rng.choice(old, nd - nd // 4), any_pair(nd // 4)])
    i = np.concatenate([any_pair(ni - ni // 4 - ni // 8), rng.choice(old, ni // 4)])
    i = np.concatenate([i, rng.choice(i, ni - len(i)) if ni > len(i) else i[:0]])  # repeats
    rng.shuffle(i)
    iw = ((i * np.uint64(2654435761)) % np.uint64(1000) + np.uint64(1)).astype(np.float32)  # (equal for repeats)
    hi = lambda p: (p >> np.uint64(32)).astype(np.uint32)
    lo = lambda p: (p & np.uint64(0xffffffff)).astype(np.uint32)
    assert (len(d), len(i)) == (nd, ni)
    Y = cuda.Graph(x)
    db = cuda.DeviceBatch(Y, lvg.HostBatch(hi(d), lo(d), np.ones(nd, np.float32), hi(i), lo(i), iw))
    Y.apply_batch(db)

    gone = np.intersect1d(d, old)
    new, first = np.unique(i, return_index=True)
    fresh = ~np.isin(new, old)
    new, first = new[fresh], first[fresh]
    stay = ~np.isin(old, gone)
    keys = np.concatenate([old[stay], new])
    order = np.argsort(keys, kind="stable")
    y = Y.download()
    assert np.array_equal(_pairs(y), keys[order])
    assert np.array_equal(y.weights, np.concatenate([x.weights[stay], iw[first]])[order])
    assert Y.size == len(keys) and Y.order == int(y.exists.sum())
    t = db.download()
    assert np.array_equal(t.del_src.astype(np.uint64) << np.uint64(32) | t.del_dst, gone)
    assert np.array_equal(t.ins_src.astype(np.uint64) << np.uint64(32) | t.ins_dst, new)
    assert np.array_equal(t.ins_w, iw[first])
