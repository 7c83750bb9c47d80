"""The work that users of louvain-gb300 have it do, as timed cases.

Each case names a workload by its sizes; ``prepare`` builds what a program has
in hand before the call (graphs, batches and prior states in HBM or in pinned
host memory, from the seed alone), ``run`` makes one pass through the public
entry points and returns the whole result. Graphs are the two families of the
benchmark's workloads: planted partitions (equal blocks, vertex ids 1..n) and
R-MAT (a/b/c = 0.57/0.19/0.19), with unit weights or small interaction counts.

Two runs of a static call in the default (asynchronous) mode end in different
clusterings of the same quality, so the static workloads ask for deterministic
mode, which runs the same kernels with the moves of a colour class applied
together. The dynamic methods start from a clustering and move few vertices:
they run in the default mode where the outcome is steady.
"""
from __future__ import annotations

import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "louvain-communities-openmp-dynamic_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import lvg  # noqa: E402

METHODS = {"naive": lvg.METHOD_NAIVE, "delta": lvg.METHOD_DELTA, "frontier": lvg.METHOD_FRONTIER}


def listed():
    """The workloads, smallest to largest range of each entry point."""
    return [
        # clustering a graph of the unit tests' size, where launches and synchronisations are the cost
        {"name": "static_pp2k", "kind": "static", "family": "pp", "n": 2048, "block": 128, "degree": 16.0,
         "p_in": 0.8, "weights": "unit"},
        # the plain static run of the first benchmark configuration (131072 vertices in 1024 communities)
        {"name": "static_pp131k", "kind": "static", "family": "pp", "n": 131072, "block": 128, "degree": 16.0,
         "p_in": 0.8, "weights": "unit"},
        # a power-law graph with interaction counts as edge weights (the weighted kernels)
        {"name": "static_rmat18_counts", "kind": "static", "family": "rmat", "scale": 18, "degree": 16.0,
         "weights": "counts"},
        # clustering one graph of the serving workload from scratch (its admission), middle of the range
        {"name": "static_rmat20", "kind": "static", "family": "rmat", "scale": 20, "degree": 16.0,
         "weights": "unit"},
        # the largest plain clustering: 8.4M vertices, 2.6e8 directed edges
        {"name": "static_rmat23", "kind": "static", "family": "rmat", "scale": 23, "degree": 16.0,
         "weights": "unit"},
        # many uneven planted partitions packed into one union (the batched workload's distribution)
        {"name": "union_96", "kind": "union", "graphs": 96, "least": 1000, "most": 256000},
        # the drop-in dynamic-frontier call on host arrays, default options, a small batch on the first
        # configuration's graph
        {"name": "frontier_host_pp131k", "kind": "host", "family": "pp", "n": 131072, "block": 128, "degree": 16.0,
         "p_in": 0.8, "weights": "unit", "method": "frontier", "fraction": 1e-4, "deterministic": False},
        # the drop-in delta-screening call on host arrays, a larger batch
        {"name": "delta_host_rmat21", "kind": "host", "family": "rmat", "scale": 21, "degree": 16.0,
         "weights": "unit", "method": "delta", "fraction": 1e-3, "deterministic": False},
        # naive-dynamic on state kept in HBM: every vertex of a power-law graph looked at again
        {"name": "naive_rmat22", "kind": "stream", "family": "rmat", "scale": 22, "degree": 16.0,
         "weights": "unit", "method": "naive", "fraction": 1e-3, "steps": 1, "deterministic": False},
        # a temporal stream of small insertion-mostly batches, each applied in HBM and followed by
        # dynamic frontier from the previous result (default options)
        {"name": "stream_pp1m", "kind": "stream", "family": "pp", "n": 1000003, "block": 1000, "degree": 32.0,
         "p_in": 0.85, "weights": "unit", "method": "frontier", "fraction": 1e-5, "steps": 4,
         "deterministic": False},
        # the headline: one batch of 1e-4 of the edges on R-MAT scale 24, applied and followed by dynamic
        # frontier, then undone the same way
        {"name": "stream_rmat24", "kind": "stream", "family": "rmat", "scale": 24, "degree": 16.0,
         "weights": "unit", "method": "frontier", "fraction": 1e-4, "steps": 1, "deterministic": True},
        # the quality check after a clustering: FP64 modularity of a host membership
        {"name": "modularity_rmat22", "kind": "modularity", "family": "rmat", "scale": 22, "degree": 16.0,
         "weights": "unit"},
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["static", "static", "static", "union", "host", "host", "stream", "stream", "modularity"])
    if kind == "union":
        return {"kind": kind, "graphs": rng.randint(8, 96), "least": rng.randint(500, 2000),
                "most": rng.randint(20000, 256000)}
    family = rng.choice(["pp", "rmat"])
    c = {"kind": kind, "family": family, "weights": "unit"}
    if family == "pp":
        top = 1000003 if kind == "stream" else 300001
        c.update(n=int(_log_uniform(rng, 1501, top)), block=rng.randint(60, 260),
                 degree=round(rng.uniform(8.0, 32.0), 2), p_in=round(rng.uniform(0.75, 0.9), 3))
    else:
        c.update(scale=rng.randint(14, 22), degree=round(rng.uniform(6.0, 20.0), 2))
    if kind == "static" and (c.get("n", 0) or c.get("scale", 0) <= 19) and rng.random() < 0.4:
        c["weights"] = "counts"
    if kind in ("host", "stream"):
        c.update(method=rng.choice(["naive", "delta", "frontier", "frontier"]),
                 fraction=float("%.3g" % _log_uniform(rng, 1e-5, 3e-3)))
        c["deterministic"] = family == "rmat" or c["fraction"] > 1e-4
    if kind == "stream":
        c["steps"] = rng.randint(1, 3)
    return c


# ------------------------------------------------------------------ inputs

def _mix(x):
    """A 64-bit hash of each element (splitmix64's finaliser)."""
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _graph(case, seed):
    """The case's graph in HBM; seeded. Counts: each undirected edge weighs 1..16."""
    if case["family"] == "pp":
        g = lvg.Graph.planted_partition(case["n"], case["block"], case["degree"], case["p_in"], seed)
    else:
        g = lvg.Graph.rmat(case["scale"], case["degree"], seed=seed)
    if case["weights"] == "unit":
        return g
    h = g.download()
    g.close()
    u = np.repeat(np.arange(h.span, dtype=np.uint64), np.diff(h.offsets).astype(np.int64))
    v = h.keys.astype(np.uint64)
    pair = np.minimum(u, v) << np.uint64(32) | np.maximum(u, v)
    w = (np.uint64(1) + _mix(pair + np.uint64(seed)) % np.uint64(16)).astype(np.float32)
    return lvg.Graph(lvg.HostGraph(h.offsets, h.keys, w, h.exists))


def _pinned(span):
    """Pinned host arrays for a state or a result: membership, vertex and community weights."""
    m = torch.empty(span, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    return m, *(torch.empty(span, dtype=torch.float64, pin_memory=True).numpy() for _ in range(2))


def _batch(g, case, seed):
    """A batch of `fraction` of the directed edges (a fifth deletions), tidied and applied to g."""
    entries = max(10, int(case["fraction"] * g.size))
    deletions = entries // 5
    drawn = lvg.DeviceBatch.generate(g, deletions, entries - deletions, seed=seed)
    raw = drawn.download()
    drawn.close()
    return g.apply_batch(raw)


def _inverse(b):
    """The batch that undoes a tidied batch (unit weights)."""
    return lvg.HostBatch(b.ins_src, b.ins_dst, b.ins_w, b.del_src, b.del_dst, b.del_w)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "union":
        n = case["graphs"]
        rng = np.random.default_rng(n)  # the graphs' sizes are the case's, their edges the seed's
        sizes = np.exp(rng.uniform(np.log(case["least"]), np.log(case["most"]), n)).astype(np.int64)
        degrees, p_in = rng.uniform(8, 32, n), rng.uniform(0.6, 0.9, n)
        graphs = [lvg.Graph.planted_partition(int(sizes[i]), 128, float(degrees[i]), float(p_in[i]), seed + i)
                  for i in range(n)]
        s["graph"] = lvg.Graph.union(graphs)
        for g in graphs:
            g.close()
        s["options"] = lvg.LouvainOptions(deterministic=True)
        return s
    g = s["graph"] = _graph(case, seed)
    if kind == "static":
        s["options"] = lvg.LouvainOptions(deterministic=True)
        s["out"] = _pinned(g.span)
        return s
    # a prior clustering, the same for the same seed
    prior = lvg.State(g)
    lvg.run_resident(g, lvg.METHOD_STATIC, None, None, prior, lvg.LouvainOptions(deterministic=True))
    if kind == "modularity":
        s["membership"] = prior.membership()
        prior.close()
        return s
    s["options"] = lvg.LouvainOptions(deterministic=case["deterministic"])
    s["out"] = _pinned(g.span)
    if kind == "host":
        s["prior"] = _pinned(g.span)
        for a, b in zip(s["prior"], prior.get()):
            a[:] = b
        prior.close()
        s["batch"] = _batch(g, case, seed + 1)
        return s
    s["prior"], s["states"] = prior, [lvg.State(g), lvg.State(g)]
    batches = [_batch(g, case, seed + 1 + i) for i in range(case["steps"])]
    undo = [_inverse(b) for b in reversed(batches)]
    for b in undo:
        g.apply_batch(b)
    s["batches"] = batches + undo
    s["device_batch"] = lvg.DeviceBatch(g, batches[0])
    return s


# ------------------------------------------------------------------ one pass

def _result(m, vw, cw, **scalars):
    return {"membership": m.view(np.int32), "vertexWeight": vw, "communityWeight": cw, **scalars}


def run(state):
    case, g = state["case"], state["graph"]
    kind = case["kind"]
    if kind == "static":
        r = lvg.louvain_static(g, state["options"], out_buffers=state["out"])
        return _result(r.membership, r.vertexWeight, r.communityWeight, iterations=r.iterations, passes=r.passes,
                       affected=r.affectedVertices)
    if kind == "union":
        rs = lvg.louvain_static_union(g, state["options"])
        span = sum(len(r.membership) for r in rs)
        whole = rs[0]  # the graphs' results lie back to back in three arrays
        return _result(whole.membership.base[:span], whole.vertexWeight.base[:span],
                       whole.communityWeight.base[:span], iterations=np.array([r.iterations for r in rs]),
                       passes=np.array([r.passes for r in rs]))
    if kind == "modularity":
        return {"modularity": g.modularity(state["membership"])}
    if kind == "host":
        call = {"naive": lvg.louvain_naive_dynamic, "delta": lvg.louvain_dynamic_delta_screening,
                "frontier": lvg.louvain_dynamic_frontier}[case["method"]]
        r = call(g, state["batch"], *state["prior"], state["options"], out_buffers=state["out"])
        return _result(r.membership, r.vertexWeight, r.communityWeight)
    # stream: each batch is uploaded, tidied and applied in HBM, and answered from the previous result;
    # then the batches are undone in reverse order the same way, so that a pass leaves the graph as it was
    method, batch, prior = METHODS[case["method"]], state["device_batch"], state["prior"]
    for i, b in enumerate(state["batches"]):
        batch.set(b)
        g.apply_batch(batch)
        out = state["states"][i % 2]
        lvg.run_resident(g, method, batch, prior, out, state["options"])
        prior = out
    m, vw, cw = state["out"]
    if lvg.load_library().lvg_state_get(prior.h, m.ctypes.data, vw.ctypes.data, cw.ctypes.data) != lvg.LVG_OK:
        raise RuntimeError("lvg_state_get failed")
    return _result(m, vw, cw)


# ------------------------------------------------------------------ what a pass cannot do without

def _sizes(case):
    """(vertices, directed edges) of the case's graph, about."""
    n = case["n"] if case["family"] == "pp" else 1 << case["scale"]
    return n, n * case["degree"] * (1.0 if case["family"] == "pp" else 2.0)


def work(case):
    """Inputs read once and outputs written once: a CSR is 8 bytes an edge (4 where
    weights are known to be one) and 12 a vertex, a state 20 bytes a vertex, a batch
    entry 12 bytes."""
    kind = case["kind"]
    if kind == "union":
        n = case["graphs"] * (case["most"] - case["least"]) / np.log(case["most"] / case["least"])
        return {"bytes": float(n * (20 * 4 + 12 + 20)), "flops": 0.0}
    n, x = _sizes(case)
    csr = x * (8 if case["weights"] == "counts" else 4) + 12 * n
    if kind == "static":
        return {"bytes": csr + 20 * n, "flops": 0.0}
    if kind == "modularity":
        return {"bytes": csr + 4 * n, "flops": 0.0}
    entries = max(10.0, case["fraction"] * x)
    scan = csr if case["method"] == "naive" else entries * 4 * case["degree"]
    steps = 2 * case["steps"] if kind == "stream" else 1
    return {"bytes": steps * (scan + 12 * entries) + 40 * n, "flops": 0.0}


# ------------------------------------------------------------------ 64-bit values

def exact(case, seed):
    """The vertex weights are the weighted degrees of the graph that the pass leaves (a
    stream leaves the one it began with), modularity its definition; the other outputs
    are the algorithm's decisions."""
    if case["kind"] == "union" or _sizes(case)[1] > 1.5e8:
        return None
    s = prepare(case, seed)
    h = s["graph"].download()
    offsets = torch.from_numpy(h.offsets.astype(np.int64)).cuda()
    row = torch.repeat_interleave(torch.arange(h.span, device="cuda"), offsets.diff())
    w = torch.from_numpy(h.weights).cuda().double()
    degree = torch.zeros(h.span, dtype=torch.float64, device="cuda").index_add_(0, row, w)
    if case["kind"] == "modularity":
        m = torch.from_numpy(s["membership"].astype(np.int64)).cuda()
        key = torch.from_numpy(h.keys.astype(np.int64)).cuda()
        inside = w[m[row] == m[key]].sum()
        total = torch.zeros(h.span, dtype=torch.float64, device="cuda").index_add_(0, m, degree)
        M2 = w.sum()
        return {"modularity": float(inside / M2 - total.square().sum() / (M2 * M2))}
    return {"membership": None, "vertexWeight": degree.cpu().numpy(), "communityWeight": None}
