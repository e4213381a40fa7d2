"""Workloads of the Louvain engine, for timing it through its public entry points.

A case is a dict of plain values.  Its "path" says which entry point it goes through:

  louvain    Graph.louvain on a graph that is resident on the device
  batch      Batch.run on many graphs packed as one union
  upload     Context.graph_from_csr from page-locked host arrays, then Graph.louvain
  coarsen    Graph.coarsen by a given assignment, the new graph's CSR read back
  modularity Graph.modularity of a given assignment
  sweep      mg_local_move_noalloc, one local-move sweep over device arrays

Full runs and batches work on the engine's own seeded generators (SBM, R-MAT, Chung-Lu), the
others on graphs made here with torch.  A program keeps one context for all its graphs, so the
module does too.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

mg = importlib.import_module("mg-alphagcd_b200")

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = mg.Context(0)
    return _ctx


def listed():
    return [
        # An interactive call on a small graph (the smallest of the batched workload's range):
        # launches, synchronisations and host work are the whole cost.
        dict(name="louvain_sbm_1k", path="louvain", kind="sbm", n=1013, blocks=4, degree=8.0, intra=0.8, version=2,
             precision="fp64"),
        # The plain-Louvain workload of the benchmark.
        dict(name="louvain_sbm_64k", path="louvain", kind="sbm", n=65536, blocks=64, degree=16.0, intra=0.8,
             version=2, precision="fp64"),
        # A skewed graph of ordinary size under the version-1 rule.
        dict(name="louvain_rmat_18_v1", path="louvain", kind="rmat", scale=18, edge_factor=16, version=1,
             precision="fp64"),
        # An ordinary large graph with exact integer gains.
        dict(name="louvain_rmat_21_int64", path="louvain", kind="rmat", scale=21, edge_factor=16, version=2,
             precision="int64"),
        # The headline workload: the largest graph, R-MAT scale 24 to convergence.
        dict(name="louvain_rmat_24", path="louvain", kind="rmat", scale=24, edge_factor=16, version=2,
             precision="fp64"),
        # Real weights (lognormal, float) on a power-law graph, FP32 gains; a ragged vertex count.
        dict(name="louvain_chunglu_f32", path="louvain", kind="chunglu", n=300007, degree=20.0, max_degree=20000.0,
             lognormal=True, version=2, precision="fp32"),
        # A packed batch of small graphs, as a server forms it: latency of many short phases.
        dict(name="batch_sbm_48", path="batch", graphs=48, n_min=1000, n_max=8000),
        # The batched workload of the benchmark at an eighth of its graph count.
        dict(name="batch_sbm_512", path="batch", graphs=512, n_min=1000, n_max=200000),
        # End to end from host memory: a graph streamed in and clustered once.
        dict(name="upload_run_1m", path="upload", n=1000003, entries=12000000, blocks=1000, skew=1.0, weights="unit"),
        # One coarsening step of a caller's own loop, real weights, with the new level read back.
        dict(name="coarsen_30k_f64", path="coarsen", n=30011, entries=600000, blocks=200, skew=1.5, weights="f64",
             groups=3000),
        # The quality of a partition that another program found.
        dict(name="modularity_2m", path="modularity", n=2000003, entries=32000000, blocks=5000, skew=1.5,
             weights="unit", groups=100000),
        # One sweep on device arrays for a caller that cannot allocate; integer weights, skewed degrees.
        dict(name="sweep_500k", path="sweep", n=500009, entries=10000000, blocks=500, skew=2.0, weights="int",
             groups=100000, version=2, up=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["louvain", "louvain", "louvain", "batch", "upload", "coarsen", "modularity", "sweep"])
    if path == "louvain":
        kind = rng.choice(["sbm", "rmat", "chunglu"])
        c = dict(path=path, kind=kind, version=rng.choice([2, 2, 1]), precision=rng.choice(["fp64", "fp64", "int64"]))
        if kind == "sbm":
            c.update(n=_log(rng, 1000, 1000000), blocks=rng.randint(4, 256), degree=round(rng.uniform(8, 32), 3),
                     intra=round(rng.uniform(0.7, 0.9), 3))
        elif kind == "rmat":
            c.update(scale=rng.randint(10, 22), edge_factor=rng.randint(8, 20))
        else:
            n = _log(rng, 5000, 1000000)
            c.update(n=n, degree=round(rng.uniform(8, 24), 3), max_degree=float(max(100, n // 16)), lognormal=False)
        return c
    if path == "batch":
        n_max = _log(rng, 4000, 200000)
        return dict(path=path, graphs=_log(rng, 8, 256), n_min=1000, n_max=n_max)
    n = _log(rng, 1000, 2000000)
    entries = n * rng.randint(8, 24)
    c = dict(path=path, n=n, entries=entries, blocks=max(2, _log(rng, n / 1000 + 2, n / 50 + 3)),
             skew=round(rng.uniform(1.0, 2.0), 3))
    if path == "upload":
        c.update(weights=rng.choice(["unit", "unit", "int"]))
        return c
    c.update(groups=max(2, _log(rng, n / 100 + 2, n / 2)))
    if path == "coarsen":
        c.update(weights=rng.choice(["unit", "int", "f64"]))
        c["entries"] = min(c["entries"], 4000000)
        c["n"] = min(c["n"], 400000)
        c["groups"] = min(c["groups"], c["n"] // 2)
    elif path == "modularity":
        c.update(weights=rng.choice(["unit", "int", "f64"]))
    else:
        c.update(weights=rng.choice(["unit", "int"]), version=rng.choice([1, 2]), up=rng.choice([0, 1]))
    return c


# ---- graphs made here: planted blocks, degrees skewed by drawing ends as n * u^skew -----------


def _graph(case, seed):
    """CSR on the device: offsets (int64), cols (int32), weights (float64 or None).  Symmetric,
    rows sorted, duplicate pairs merged, a few self-loops."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(1000003 * seed + 17)
    n, m, blocks = case["n"], case["entries"] // 2, case["blocks"]
    u = (torch.rand(m, generator=g, device=dev, dtype=torch.float64) ** case["skew"] * n).long().clamp_(0, n - 1)
    size = -(-n // blocks)
    inside = (u // size) * size + (torch.rand(m, generator=g, device=dev) * size).long()
    outside = (torch.rand(m, generator=g, device=dev, dtype=torch.float64) ** case["skew"] * n).long()
    v = torch.where(torch.rand(m, generator=g, device=dev) < 0.75, inside, outside).clamp_(0, n - 1)
    # ids without order: a random renumbering of the vertices
    name = torch.randperm(n, generator=g, device=dev)
    u, v = name[u], name[v]
    keys = torch.unique(torch.cat([u * n + v, v * n + u]))
    row, col = keys // n, keys % n
    off = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    off[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    lo, hi = torch.minimum(row, col), torch.maximum(row, col)
    h = (lo * 2654435761 + hi * 40503 + seed * 7919) % 1000003  # equal for both directions
    if case["weights"] == "unit":
        w = None
    elif case["weights"] == "int":
        w = (h % 9 + 1).double()
    else:
        w = torch.exp(h.double() / 1000003 * 4 - 2)
    return off, col.int(), w


def _groups(case, seed):
    """An assignment into case["groups"] communities, each named by one of its members as the
    engine's own sweeps do."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(7907 * seed + 5)
    n = case["n"]
    reps = torch.randperm(n, generator=g, device=dev)[: min(case["groups"], n)]
    C = reps[torch.randint(len(reps), (n,), generator=g, device=dev)]
    C[reps] = reps
    return C


def _host_csr(case, seed, pinned=False):
    off, col, w = _graph(case, seed)

    def host(t, dtype):
        t = t.cpu()
        return (t.pin_memory() if pinned else t).numpy().view(dtype)

    return host(off, np.uint64), host(col, np.uint32), None if w is None else host(w, np.float64)


def prepare(case, seed):
    path, ctx = case["path"], _context()
    if path == "louvain":
        if case["kind"] == "sbm":
            graph = ctx.generate_sbm(case["n"], case["blocks"], case["degree"], case["intra"], seed=seed)
        elif case["kind"] == "rmat":
            graph = ctx.generate_rmat(case["scale"], case["edge_factor"], seed=seed)
        else:
            graph = ctx.generate_chunglu(case["n"], 2.1, case["degree"], case["max_degree"],
                                         lognormal=case["lognormal"], seed=seed)
        return dict(path=path, graph=graph, version=case["version"], precision=case["precision"])
    if path == "batch":
        # the sizes are the case's (the benchmark's draw), the graphs the seed's
        params = mg.draw_sbm_params(case["graphs"], (case["n_min"], case["n_max"]), (4, 256), (8.0, 32.0), (0.7, 0.9),
                                    seed=4)
        for i, p in enumerate(params):
            p["seed"] = 100003 * seed + i
        return dict(path=path, batch=ctx.batch_generate_sbm(params))
    if path == "upload":
        off, col, w = _host_csr(case, seed, pinned=True)
        return dict(path=path, ctx=ctx, n=case["n"], off=off, col=col, w=w)
    if path in ("coarsen", "modularity"):
        off, col, w = _host_csr(case, seed)
        C = _groups(case, seed).cpu().numpy().astype(np.uint32)
        state = dict(path=path, graph=ctx.graph_from_csr(case["n"], off, col, w), C=C)
        if path == "coarsen":  # buffers that hold any coarsening of the graph
            state.update(off=np.zeros(case["groups"] + 1, np.uint64), col=np.zeros(case["entries"], np.uint32),
                         w=np.zeros(case["entries"]))
        return state
    # one sweep: the caller's own device arrays
    off, col, w = _graph(case, seed)
    n = case["n"]
    weights = torch.ones(len(col), dtype=torch.float64, device=col.device) if w is None else w
    row = torch.repeat_interleave(torch.arange(n, device=col.device), off[1:] - off[:-1])
    k = torch.zeros(n, dtype=torch.float64, device=col.device).index_add_(0, row, weights)
    C = _groups(case, seed)
    sigma = torch.zeros(n, dtype=torch.float64, device=col.device).index_add_(0, C, k)
    return dict(path=path, n=n, off=off.int(), col=col, w=w, mass=float(weights.sum()), C=C.int(), sigma=sigma, k=k,
                out=torch.empty(n, dtype=torch.int32, device=col.device), version=case["version"], up=case["up"])


def _result(r):
    # the tables have a row per iteration and per level: into arrays of one size for every graph
    trace, sizes = np.zeros((1024, 4)), np.zeros(64, np.uint32)
    trace[: len(r["trace"])] = r["trace"]
    sizes[: len(r["level_sizes"])] = r["level_sizes"]
    return dict(assignment=r["assignment"], level_sizes=sizes, trace=trace, modularity=r["modularity"])


def run(state):
    path, L = state["path"], mg.lib()
    if path == "louvain":
        return _result(state["graph"].louvain(version=state["version"], precision=state["precision"]))
    if path == "batch":
        r = state["batch"].run()
        return dict(modularity=r["graphs"]["modularity"], communities=r["graphs"]["communities"],
                    iterations=r["graphs"]["iterations"].astype(np.int64), assignment=np.concatenate(r["assignments"]))
    if path == "upload":
        graph = state["ctx"].graph_from_csr(state["n"], state["off"], state["col"], state["w"])
        out = _result(graph.louvain())
        graph.close()
        return out
    if path == "modularity":
        return state["graph"].modularity(state["C"])
    if path == "coarsen":
        dense, level = state["graph"].coarsen(state["C"])
        off, col, w = state["off"], state["col"], state["w"]
        status = L.mg_graph_copy_csr(level.h, *(ctypes.c_void_p(a.ctypes.data) for a in (off, col, w)))
        level.close()
        if status != mg.MG_OK:
            raise mg.MGError(status, "mg_graph_copy_csr")
        return dict(dense=dense, off=off.view(np.int64), col=col, w=w)
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
    status = L.mg_local_move_noalloc(
        ctypes.c_uint32(state["n"]), p(state["off"]), p(state["col"]), p(state["w"]), ctypes.c_double(state["mass"]),
        p(state["C"]), p(state["sigma"]), p(state["k"]), p(state["out"]), state["version"], state["up"],
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if status != mg.MG_OK:
        raise mg.MGError(status, L.mg_last_error(None).decode())
    return state["out"]


def work(case):
    """The graph (and assignment) read once and the result written once; one gain per entry for
    a sweep, one compare and add per entry otherwise."""
    path = case["path"]
    if path == "louvain":
        if case["kind"] == "rmat":
            n = 1 << case["scale"]
            entries = 2 * case["edge_factor"] << case["scale"]
        else:
            n, entries = case["n"], int(case["n"] * case["degree"])
        wide = 4 if case.get("lognormal") else 0
        return dict(bytes=entries * (4 + wide) + 8 * n, flops=8 * entries)
    if path == "batch":
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])  # of a log-uniform draw
        n, entries = case["graphs"] * mean, case["graphs"] * mean * 20
        return dict(bytes=4 * entries + 8 * n, flops=8 * entries)
    n, entries = case["n"], case["entries"]
    wide = 0 if case["weights"] == "unit" else 8
    if path == "upload":
        return dict(bytes=entries * (4 + wide) + 12 * n, flops=8 * entries)
    if path == "coarsen":
        return dict(bytes=entries * (4 + wide) + 8 * n + 12 * entries, flops=entries)
    if path == "modularity":
        return dict(bytes=entries * (4 + wide) + 8 * n, flops=2 * entries)
    return dict(bytes=entries * (4 + wide) + 28 * n, flops=8 * entries)


def exact(case, seed):
    """What run() computes, in 64 bits with torch.  Full runs and batches follow a path of many
    accept / reject decisions and a sweep returns whole numbers alone: no value here."""
    path = case["path"]
    if path not in ("modularity", "coarsen"):
        return None
    off, col, w = _graph(case, seed)
    C = _groups(case, seed)
    n = case["n"]
    col = col.long()
    w = torch.ones(len(col), dtype=torch.float64, device=col.device) if w is None else w
    row = torch.repeat_interleave(torch.arange(n, device=col.device), off[1:] - off[:-1])
    if path == "modularity":
        mass = w.sum()
        inner = w[C[row] == C[col]].sum()
        sigma = torch.zeros(n, dtype=torch.float64, device=col.device).index_add_(0, C[row], w)
        return float(inner / mass - (sigma / mass).square().sum())
    used = torch.unique(C)
    dense = torch.searchsorted(used, C)
    nn = len(used)
    keys, back = torch.unique(dense[row] * nn + dense[col], return_inverse=True)
    sums = torch.zeros(len(keys), dtype=torch.float64, device=col.device).index_add_(0, back, w)
    new_off = torch.zeros(nn + 1, dtype=torch.int64, device=col.device)
    new_off[1:] = torch.cumsum(torch.bincount(keys // nn, minlength=nn), 0)
    out = dict(dense=dense.int().cpu().numpy().view(np.uint32), off=new_off.cpu().numpy(),
               col=np.zeros(case["entries"], np.uint32), w=np.zeros(case["entries"]))
    out["col"][: len(keys)] = (keys % nn).cpu().numpy()
    out["w"][: len(keys)] = sums.cpu().numpy()
    return out
