"""Building a hub's table at the limit of 16384 neighbour communities (more:
the hub keeps scanning its edges), from scratch tables that hold a hub's whole
degree twice and from those cut to 65536 slots: deterministic results with
tables equal those without, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [20000, 70000])
@pytest.mark.parametrize("communities", [1, 16383, 16384, 19999])
def test_hub_of_many_communities(cuda, lvg, leaves, communities):
    # (one more community is the pair's)
    ids = np.arange(2, leaves + 2)  # vertex 1 is the hub; the last two ids are a pair beside the star
    a = np.concatenate([np.full(leaves, 1), [leaves + 2]])
    b = np.concatenate([ids, [leaves + 3]])
    x = lvg.csr_from_edges(leaves + 3, np.concatenate([a, b]).astype(np.uint32),
                           np.concatenate([b, a]).astype(np.uint32))
    Y = cuda.Graph(x)
    q = np.arange(x.span, dtype=np.uint32)
    q[ids] = 2 + (ids - 2) % communities
    q[leaves + 3] = leaves + 2
    deg = np.diff(x.offsets).astype(np.float64)
    u, v = np.uint32(1), np.uint32(leaves + 2)  # the batch: an edge between the hub and the pair, marks both
    e = np.empty(0, np.uint32)
    hb = lvg.HostBatch(e, e, np.empty(0, np.float32), np.array([u, v]), np.array([v, u]), np.ones(2, np.float32))
    db = cuda.DeviceBatch(Y, hb)
    Y.apply_batch(db)
    o = cuda.LouvainOptions(deterministic=True)
    prior = cuda.State(Y)
    prior.set(q, deg, np.bincount(q, weights=deg, minlength=x.span))
    outs = []
    for tables in (0, 1, 1):  # scans; tables built; tables from the prior's cache
        cuda.set_tuning(Y, hub_tables=tables)
        out = cuda.State(Y)
        info = cuda.run_resident(Y, cuda.METHOD_FRONTIER, db, prior, out, o)
        outs.append((out.get(), info["iterations"], info["passes"], Y.stats()))
    assert outs[0][3]["hub_table_slots"] == 0
    for r, i, p, st in outs[1:]:
        assert (st["hub_table_slots"] > 0) == (communities + 1 <= 16384)
        assert (i, p) == outs[0][1:3]
        assert all(np.array_equal(m, n) for m, n in zip(r, outs[0][0]))
