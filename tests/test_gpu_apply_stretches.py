"""A batch large enough that each warp of the apply takes stretches of several
hundred entries: rows longer than a stretch (most of it moved by one shift),
stretches of many short rows, rows that grow into the pool, deletions of absent
and insertions of present edges, repeated entries. The updated graph and the
tidied batch are compared with numpy's set operations: integers and weights
copied, so equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(x):
    row = np.repeat(np.arange(x.span, dtype=np.uint64), np.diff(x.offsets).astype(np.int64))
    return row << np.uint64(32) | x.keys.astype(np.uint64)


@pytest.mark.parametrize("kind", ["both", "deletions", "insertions"])
def test_long_stretches(cuda, lvg, kind):
    rng = np.random.default_rng(11)
    x = lvg.rmat(18, 16, seed=4)
    x.weights[:] = rng.integers(1, 100, len(x.weights)).astype(np.float32)
    old = _rows(x)
    d = np.concatenate([rng.choice(old, 30000), rng.choice(old, 100).repeat(2),
                        rng.integers(1, x.span, 1000).astype(np.uint64) << np.uint64(32) | np.uint64(7)])
    i = np.concatenate([rng.integers(1, x.span, 30000).astype(np.uint64) << np.uint64(32)
                        | rng.integers(1, x.span, 30000).astype(np.uint64),
                        rng.choice(old, 500),  # present
                        (np.uint64(3) << np.uint64(32)) | np.arange(100000, 120000, dtype=np.uint64)])  # a row that grows
    i = np.concatenate([i, i[:200]])
    none = np.empty(0, np.uint64)
    d, i = (none if kind == "insertions" else d), (none if kind == "deletions" else i)
    iw = ((i * np.uint64(2654435761)) % np.uint64(1000) + np.uint64(1)).astype(np.float32)  # (equal for repeats)
    hi = lambda p: (p >> np.uint64(32)).astype(np.uint32)
    lo = lambda p: (p & np.uint64(0xffffffff)).astype(np.uint32)
    Y = cuda.Graph(x)
    db = cuda.DeviceBatch(Y, lvg.HostBatch(hi(d), lo(d), np.ones(len(d), np.float32), hi(i), lo(i), iw))
    Y.apply_batch(db)

    gone = np.intersect1d(d, old)
    new, first = np.unique(i, return_index=True)
    fresh = ~np.isin(new, old)
    new, first = new[fresh], first[fresh]
    stay = ~np.isin(old, gone)
    keys = np.concatenate([old[stay], new])
    order = np.argsort(keys, kind="stable")
    y = Y.download()
    assert np.array_equal(_rows(y), keys[order])
    assert np.array_equal(y.weights, np.concatenate([x.weights[stay], iw[first]])[order])
    t = db.download()
    assert np.array_equal(t.del_src.astype(np.uint64) << np.uint64(32) | t.del_dst, gone)
    assert np.array_equal(t.ins_src.astype(np.uint64) << np.uint64(32) | t.ins_dst, new)
    assert np.array_equal(t.ins_w, iw[first])
