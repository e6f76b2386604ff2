"""Measured cases: what a user of the engine has it do, through the public
entry points of python/lvb200.py (the binding of include/louvain_b200.h).

  run          Engine.run_device: a whole Louvain run, CSR and result in device memory
  host_run     Engine.run: the same on a host graph, assignment read back
  phases       Engine.load, then phase_move / phase_aggregate until the run ends
               and assignment(): the loop of the command line program
  batch        Engine.batch_run_device: many graphs as one union
  serve        Server: requests queued, every result polled
  csr          lv_csr_from_edges_device: the reader's CSR of an edge list
  communities  Engine.communities: the listing of a finished run
  modularity   Engine.modularity: Q of a given partition

Graph shapes are those of the benchmark and the tests: the banded FEM-like
matrix, the planted power-law graph, LFR-style graphs, R-MAT, batches of
stochastic-block-model graphs.  Kernel variants are the engine's defaults
(no autotuning), as in the command line program.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "louvain-community-detection_b200", "python"))

import lvb200  # noqa: E402
import lvgen  # noqa: E402

MIN_GAIN = 1e-6
SERVE_BUDGET = 12 << 30


def listed():
    return [
        # the smallest request of the served workload: host waits and launches
        dict(name="run_lfr_1k", op="run", graph="lfr", n=1000, mu=0.3, weighted=False,
             rule="py", gain="fp32"),
        # the reference's own test matrix (a banded stiffness matrix), real weights,
        # from a host graph with the assignment read back
        dict(name="host_run_banded", op="host_run", graph="banded", n=4884, mu=0.0,
             weighted=True, rule="py", gain="fp32"),
        # the command line program's loop on an ordinary graph of odd size
        dict(name="phases_lfr_100k", op="phases", graph="lfr", n=100_003, mu=0.2,
             weighted=True, rule="py", gain="fp32"),
        # the benchmark's headline workload
        dict(name="run_powerlaw_335k", op="run", graph="powerlaw", n=334_863, mu=0.3,
             weighted=False, rule="py", gain="fp32"),
        # a weighted graph of a million vertices under the reference CUDA rule
        dict(name="run_lfr_1m_cuda_rule", op="run", graph="lfr", n=1_000_003, mu=0.4,
             weighted=True, rule="cuda", gain="fp32"),
        # FP64 gains (equal to the reference script) on a skewed graph with hubs
        dict(name="run_rmat20_fp64", op="run", graph="rmat", n=1 << 20, mu=0.0,
             weighted=False, rule="py", gain="fp64"),
        # the benchmark's largest graph, far beyond the L2
        dict(name="run_rmat24", op="run", graph="rmat", n=1 << 24, mu=0.0,
             weighted=False, rule="py", gain="fp32"),
        # many small graphs in one union
        dict(name="batch_sbm_512", op="batch", graphs=512, hi=65_536, rule="py",
             gain="fp32"),
        # requests of mixed sizes through the server's lanes
        dict(name="serve_48", op="serve", graphs=48, hi=200_000, rule="py", gain="fp32"),
        # ingest: the CSR of a weighted edge list in random file order
        dict(name="csr_lfr_2m", op="csr", graph="lfr", n=2_000_003, mu=0.3, weighted=True,
             edges=12_000_001),
        # output: the community listing of a finished run
        dict(name="communities_lfr_1m", op="communities", graph="lfr", n=1_000_003, mu=0.2,
             weighted=False, rule="py", gain="fp32"),
        # the quality of a partition that the caller brings
        dict(name="modularity_lfr_1m", op="modularity", graph="lfr", n=1_000_003, mu=0.3,
             weighted=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def draw(rng):
    op = rng.choice(["run"] * 6 + ["host_run", "phases", "batch", "serve", "csr",
                                   "communities", "modularity"])
    opts = dict(rule=rng.choice(["py", "py", "cuda"]), gain=rng.choice(["fp32", "fp32", "fp64"]))
    if op == "batch":
        return dict(op=op, graphs=_log_uniform(rng, 16, 512), hi=_log_uniform(rng, 1024, 65_536),
                    **opts)
    if op == "serve":
        return dict(op=op, graphs=_log_uniform(rng, 4, 48), hi=_log_uniform(rng, 4000, 200_000),
                    **opts)
    graph = rng.choice(["lfr", "lfr", "rmat", "powerlaw", "banded"] if op in
                       ("run", "host_run", "phases") else ["lfr", "rmat"])
    weighted = graph != "rmat" and rng.random() < 0.5
    if graph == "lfr":
        n = _log_uniform(rng, 1000, 2_000_000)
    elif graph == "rmat":
        n = 1 << rng.randint(10, 22)
    elif graph == "powerlaw":
        n = _log_uniform(rng, 2000, 400_000)
    else:
        n, weighted = _log_uniform(rng, 1000, 20_000), True
    mu = round(rng.uniform(0.1, 0.5), 3) if graph in ("lfr", "powerlaw") else 0.0
    case = dict(op=op, graph=graph, n=n, mu=mu, weighted=weighted)
    if op == "csr":
        case["edges"] = int(n * rng.uniform(4.0, 12.0))
    elif op != "modularity":
        case.update(opts)
    return case


def _edge_weights(rows, cols, seed):
    """Weights U(0.5, 1.5), the same in both rows of an edge."""
    h = torch.minimum(rows, cols) * 0x9E3779B1 + torch.maximum(rows, cols) * 0x85EBCA6B + seed
    h = (h ^ (h >> 17)) * 0x27D4EB2F
    return ((h >> 9) & 0x7FFFFF).to(torch.float32) / float(1 << 23) + 0.5


def _graph(case, seed):
    """(n, off int64, col int32, w float32) on the device, and the planted
    communities where the shape has them."""
    kind, n = case["graph"], case["n"]
    comm = None
    if kind == "lfr":
        (n, off, col, w, _), comm = lvgen.lfr_device(n, case["mu"], seed=seed)
    elif kind == "rmat":
        n, off, col, w, _ = lvgen.rmat_device(n.bit_length() - 1, seed=seed)
    else:
        if kind == "banded":
            n, s, d, w = lvgen.banded_fem(n=n, target_entries=int(59.4 * n), seed=seed)
        else:
            n, s, d, w = lvgen.planted_powerlaw(n=n, target_edges=int(2.765 * n), mu=case["mu"],
                                                max_deg=min(550, n // 8), seed=seed,
                                                unit=not case["weighted"])
        off, col, w = lvgen.csr_from_edges(n, s, d, w)
        off = torch.from_numpy(off.view(np.int64)).cuda()
        col = torch.from_numpy(col.view(np.int32)).cuda()
        w = torch.from_numpy(w).cuda()
    if case["weighted"] and kind in ("lfr", "rmat"):
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), off[1:] - off[:-1])
        w = _edge_weights(rows, col.to(torch.int64), seed)
    return n, off, col, w, comm


def _host_graph(n, off, col, w):
    return lvb200.Graph.from_csr(n, off.cpu().numpy().view(np.uint64),
                                 col.cpu().numpy().view(np.uint32), w.cpu().numpy())


def _edges(case, seed):
    """case["edges"] lines of the graph in random order (src, dst int32, w), on
    the device; a graph with fewer edges has some lines twice, as files may."""
    n, off, col, w, _ = _graph(case, seed)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), off[1:] - off[:-1])
    up = rows < col
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    src, dst, w = rows[up].to(torch.int32), col[up], w[up]
    p = torch.randperm(src.numel(), generator=gen, device="cuda")
    p = p.repeat(-(-case["edges"] // src.numel()))[:case["edges"]]
    return n, src[p].contiguous(), dst[p].contiguous(), w[p].contiguous()


def _sbm_union(case, seed):
    """Block-diagonal union of SBM graphs whose sizes belong to the case; the
    seed relabels every graph's vertices and draws the weights U(0.5, 1.5)."""
    goff, off, col, _, _ = lvgen.sbm_batch_device(case["graphs"], seed=0, hi=case["hi"])
    n = int(goff[-1])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    sizes = torch.from_numpy(np.diff(goff.astype(np.int64))).cuda()
    gid = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), sizes)
    key = gid + torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    new = torch.empty(n, dtype=torch.int64, device="cuda")
    new[torch.argsort(key)] = torch.arange(n, device="cuda")
    rows = torch.repeat_interleave(new, off[1:] - off[:-1])
    col = new[col.to(torch.int64)]
    rows, order = torch.sort(rows, stable=True)
    col = col[order]
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return goff, off, col.to(torch.int32), _edge_weights(rows, col, seed)


def _requests(case, seed):
    """Host graphs of mixed kinds, as the server gets them; their log-uniform
    sizes belong to the case, the graphs to the seed."""
    rng = np.random.default_rng(case["graphs"])
    out = []
    for i in range(case["graphs"]):
        n = int(np.exp(rng.uniform(np.log(1000), np.log(case["hi"]))))
        if i % 2:
            g = lvgen.rmat_device(max(10, n.bit_length() - 1), seed=seed + i)
        else:
            g, _ = lvgen.lfr_device(n, float(rng.uniform(0.1, 0.5)), seed=seed + i)
        out.append((_host_graph(*g[:4]), g[0]))
    return out


def prepare(case, seed):
    op = case["op"]
    s = dict(op=op)
    opts = dict(rule=case.get("rule", "py"), gain=case.get("gain", "fp32"))
    if op == "serve":
        s["reqs"] = _requests(case, seed)
        s["server"] = lvb200.Server(MIN_GAIN, SERVE_BUDGET, lanes=4, background=True, **opts)
        return s
    if op == "csr":
        n, src, dst, w = _edges(case, seed)
        m = src.numel()
        s.update(n=n, m=m, src=src, dst=dst, w=w,
                 off=torch.empty(n + 1, dtype=torch.int64, device="cuda"),
                 col=torch.empty(2 * m, dtype=torch.int32, device="cuda"),
                 wout=torch.empty(2 * m, dtype=torch.float32, device="cuda"))
        torch.cuda.synchronize()
        return s
    s["eng"] = lvb200.Engine(**opts)
    if op == "batch":
        goff, off, col, w = _sbm_union(case, seed)
        s.update(goff=goff, off=off, col=col, w=w, n=int(goff[-1]))
        s["out"] = torch.empty(s["n"], dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        return s
    n, off, col, w, comm = _graph(case, seed)
    s["n"] = n
    if op in ("host_run", "phases"):
        s["g"] = _host_graph(n, off, col, w)
        return s
    s.update(off=off, col=col, w=w, out=torch.empty(n, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    if op == "communities":
        _run_device(s)
    elif op == "modularity":
        if comm is None:
            comm = np.random.default_rng(seed).integers(0, max(1, n // 50), n)
        s["part"] = np.ascontiguousarray(comm, dtype=np.uint32)
        s["eng"].load_device(n, col.numel(), off.data_ptr(), col.data_ptr(), w.data_ptr())
    return s


def _run_device(s):
    return s["eng"].run_device(s["n"], s["col"].numel(), s["off"].data_ptr(),
                               s["col"].data_ptr(), s["w"].data_ptr(), MIN_GAIN,
                               s["out"].data_ptr())


def _padded(values, length):
    """How many there are depends on the graph: the same length for every seed."""
    out = np.zeros(length, dtype=np.uint32)
    out[:len(values)] = values
    return out


def run(s):
    op = s["op"]
    if op == "run":
        r = _run_device(s)
        return dict(assignment=s["out"], q=r.modularity, communities=r.n_communities,
                    levels=r.n_levels, edges=r.edges_processed)
    if op == "host_run":
        r = s["eng"].run(s["g"], MIN_GAIN)
        return dict(assignment=r.assignment, q=r.modularity, communities=r.n_communities,
                    passes=_padded([level["passes"] for level in r.levels], 64))
    if op == "phases":
        e = s["eng"]
        e.load(s["g"])
        while True:
            more, q = e.phase_move(MIN_GAIN)
            if not more:
                break
            e.phase_aggregate()
        return dict(assignment=e.assignment(), q=q)
    if op == "batch":
        q, levels, _ = s["eng"].batch_run_device(s["goff"], s["n"], s["col"].numel(),
                                                 s["off"].data_ptr(), s["col"].data_ptr(),
                                                 s["w"].data_ptr(), MIN_GAIN,
                                                 s["out"].data_ptr())
        return dict(assignment=s["out"], q=q, levels=levels)
    if op == "serve":
        tickets = [s["server"].submit(g, n_vertices=n) for g, n in s["reqs"]]
        done = s["server"].drain()
        res = [done[t] for t in tickets]
        return dict(assignment=np.concatenate([r.assignment for r in res]),
                    q=np.array([r.modularity for r in res]),
                    levels=np.array([r.levels for r in res]))
    if op == "csr":
        nnz = ctypes.c_uint64()
        st = lvb200.lib().lv_csr_from_edges_device(
            s["n"], s["m"], s["src"].data_ptr(), s["dst"].data_ptr(), s["w"].data_ptr(),
            s["off"].data_ptr(), s["col"].data_ptr(), s["wout"].data_ptr(), ctypes.byref(nnz),
            None)
        if st:
            raise RuntimeError(f"lv_csr_from_edges_device: status {st}")
        return dict(off=s["off"], col=s["col"], w=s["wout"], nnz=int(nnz.value))
    if op == "communities":
        offsets, members = s["eng"].communities()
        return dict(offsets=_padded(offsets, s["n"] + 1), members=members)
    return dict(q=s["eng"].modularity(s["part"]))


def _entries(case):
    """Stored entries of the shape, nearly (duplicates are merged)."""
    if "edges" in case:
        return 2.0 * case["edges"]
    per = {"lfr": 13.0, "rmat": 30.0, "powerlaw": 5.53, "banded": 59.4}
    return per[case["graph"]] * case["n"]


def work(case):
    op = case["op"]
    if op == "batch":
        n = float(lvgen.sbm_batch_sizes(case["graphs"], 0, hi=case["hi"])[0].sum())
        e = 16.0 * n
    elif op == "serve":
        n = case["graphs"] * (case["hi"] - 1000) / math.log(case["hi"] / 1000)
        e = 20.0 * n
    else:
        n, e = float(case["n"]), _entries(case)
    graph = 8.0 * e + 8.0 * (n + 1)  # column and weight of an entry, a row's offset
    if op == "csr":  # an edge line read once, the CSR written once
        return dict(bytes=6.0 * e + graph, flops=0.0)
    if op == "communities":  # assignment in, offsets and members out
        return dict(bytes=8.0 * n, flops=0.0)
    return dict(bytes=graph + 4.0 * n, flops=0.0)


def exact(case, seed):
    """Q of a given partition and the weights of the built CSR in 64 bits.
    A run's Q belongs to the partition that the run itself finds."""
    if case["op"] == "csr":
        n, src, dst, w = (x.cpu().numpy() if torch.is_tensor(x) else x
                          for x in _edges(case, seed))
        rows = np.empty(2 * len(src), dtype=np.int32)
        rows[0::2], rows[1::2] = src, dst
        order = np.argsort(rows, kind="stable")
        return dict(off=None, col=None, w=np.abs(w.astype(np.float64))[order >> 1], nnz=None)
    if case["op"] == "modularity":
        n, off, col, w, comm = _graph(case, seed)
        if comm is None:
            comm = np.random.default_rng(seed).integers(0, max(1, n // 50), n)
        part = torch.from_numpy(np.ascontiguousarray(comm, dtype=np.int64)).cuda()
        row = torch.repeat_interleave(part, off[1:] - off[:-1])
        w = w.double()
        total = float(w.sum())
        intra = float(w[row == part[col.to(torch.int64)]].sum())
        a = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row, w)
        return dict(q=intra / total - float((a / total).square().sum()))
    return None
