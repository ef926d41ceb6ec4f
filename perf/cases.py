"""Workloads of the evolving-graph engine, each one pass through its public entry points.

A case is a dict of plain values; `kind` names the program a user writes:

  stream    a graph arrives in batches: every batch is inserted and compacted, then BFS / CC /
            SSSP continue from their previous state (pipelined, as the streaming benchmark);
  prdelta   the same with PageRank-delta, updated to a tolerance after every batch, batches
            coming from host memory;
  window    one update of a sliding window on a standing graph: the new edges are inserted and
            the programs run, then the same edges expire (deletion) and the programs run again;
  traverse  programs from scratch on a standing snapshot (BFS / CC / SSSP / SSWP);
  pagerank  normalised PageRank of a standing snapshot, FP32 compensated or FP64;
  batch     a service with several snapshots: they are loaded, eight jobs on each answer in one
            batched launch, a further 5 % of the edges arrive, the jobs answer again;
  adjoint   weighted PageRank and the gradients of a loss on its ranks;
  ingest    a graph is generated (RMAT) on the device, inserted, compacted and first traversed.

Graphs: `rmat` (graph500 quadrant probabilities; `shuffled` renames the vertices at random, as
graph500 and real data sets do, otherwise the hubs have the low ids), `uniform` random pairs, and
`lattice`, a road-like grid with a tenth of its links missing (hundreds of rounds with small
frontiers). Sizes are those of this repository's benchmark workloads and tests, and the range
between the smallest and the largest of them.
"""
import math

import numpy as np
import torch

import cytom_gb300 as cg

ALPHA = 0.85
# rounds of the iterative solves at the tolerances used here, as the benchmark workloads report
# them; they only scale work()
PRDELTA_ROUNDS, PAGERANK_ROUNDS, FORWARD_ROUNDS, ADJOINT_ROUNDS = 46, 32, 21, 86


def listed():
    return [
        # The headline of the repository's benchmark: the RMAT-22 stream of 64 batches of 2^20
        # weighted edges, three programs kept up to date.
        dict(name="stream_rmat22", kind="stream", graph="rmat", shuffled=False, scale=22, vpt=65536, batch=1 << 20,
             batches=64, weighted=True, programs="bfs,cc,sssp"),
        # The benchmark's PageRank-delta stream: RMAT-16 in 16 batches of 65,536 edges from host memory.
        dict(name="prdelta_rmat16", kind="prdelta", graph="rmat", shuffled=False, scale=16, vpt=4096, batch=65536,
             batches=16),
        # One update of a live graph: 4 M edges stand, 20,011 arrive and later expire.
        dict(name="window_rmat18", kind="window", graph="rmat", shuffled=True, scale=18, vpt=65536, edges=1 << 22,
             batch=20011, weighted=True, programs="bfs,cc,sssp"),
        # The smallest query: one BFS on a small graph, where launches and latency count.
        dict(name="bfs_rmat12", kind="traverse", graph="rmat", shuffled=False, scale=12, vpt=1024, edges=65536,
             weighted=False, programs="bfs", start=0),
        # Road-like graph: many rounds with a small frontier.
        dict(name="road_lattice18", kind="traverse", graph="lattice", shuffled=False, scale=18, vpt=65536, edges=0,
             weighted=True, programs="bfs,sssp", start=0),
        # An ordinary snapshot whose ids carry no order, every program, ragged edge count.
        dict(name="traverse_rmat20", kind="traverse", graph="rmat", shuffled=True, scale=20, vpt=65536, edges=16000003,
             weighted=True, programs="bfs,cc,sssp,sswp", start=3),
        # A large snapshot (the stream's final size times four), unweighted programs.
        dict(name="traverse_rmat24", kind="traverse", graph="rmat", shuffled=True, scale=24, vpt=65536, edges=1 << 28,
             weighted=False, programs="bfs,cc", start=0),
        # The benchmark's precision workload at a quarter of its size, both forms.
        dict(name="pagerank32_rmat24", kind="pagerank", graph="rmat", shuffled=False, scale=24, vpt=65536,
             edges=1 << 28, fp64=False),
        dict(name="pagerank64_rmat22", kind="pagerank", graph="rmat", shuffled=True, scale=22, vpt=65536,
             edges=60000007, fp64=True),
        # The benchmark's batching workload: 64 jobs over snapshots of scales 14 to 21.
        dict(name="batch64", kind="batch", lo=14, hi=21, factor=16),
        # The benchmark's differentiation workload: RMAT-20, forward solve and gradients to the host.
        dict(name="adjoint_rmat20", kind="adjoint", graph="rmat", shuffled=False, scale=20, vpt=65536, edges=1 << 24),
        # Time to the first answer of a generated graph: 50 M weighted edges in four chunks.
        dict(name="ingest_rmat22", kind="ingest", scale=22, vpt=65536, edges=50000003, chunks=4, weighted=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _some(rng, names):
    got = [x for x in names if rng.random() < 0.6]
    return ",".join(got or [rng.choice(names)])


def _vpt(rng, scale):
    top = min(16, scale)
    return 1 << rng.randint(min(top, max(8, scale - 6)), top)


def draw(rng):
    kind = rng.choice(["stream", "prdelta", "window", "traverse", "traverse", "pagerank", "batch", "adjoint", "ingest"])
    shuffled = rng.random() < 0.5
    if kind == "stream":
        scale, batch = rng.randint(16, 22), _log(rng, 1 << 13, 1 << 20)
        weighted = rng.random() < 0.7
        progs = _some(rng, ["bfs", "cc", "sssp"] if weighted else ["bfs", "cc"])
        return dict(kind=kind, graph="rmat", shuffled=shuffled, scale=scale, vpt=_vpt(rng, scale), batch=batch,
                    batches=rng.randint(4, 48), weighted=weighted, programs=progs)
    if kind == "prdelta":
        scale = rng.randint(12, 18)
        return dict(kind=kind, graph="rmat", shuffled=shuffled, scale=scale, vpt=_vpt(rng, scale),
                    batch=_log(rng, 1 << 12, 1 << 17), batches=rng.randint(3, 16))
    if kind == "window":
        scale = rng.randint(14, 20)
        weighted = rng.random() < 0.7
        progs = _some(rng, ["bfs", "cc", "sssp", "sswp"] if weighted else ["bfs", "cc"])
        return dict(kind=kind, graph=rng.choice(["rmat", "uniform"]), shuffled=shuffled, scale=scale,
                    vpt=_vpt(rng, scale), edges=_log(rng, 4 << scale, 16 << scale), batch=_log(rng, 200, 200000),
                    weighted=weighted, programs=progs)
    if kind == "traverse":
        graph = rng.choice(["rmat", "rmat", "uniform", "lattice"])
        scale = rng.randint(12, 18) if graph == "lattice" else rng.randint(10, 24)
        weighted = rng.random() < 0.6
        progs = _some(rng, ["bfs", "cc", "sssp", "sswp"] if weighted else ["bfs", "cc"])
        edges = 0 if graph == "lattice" else _log(rng, 4 << scale, 16 << scale)
        return dict(kind=kind, graph=graph, shuffled=shuffled, scale=scale, vpt=_vpt(rng, scale), edges=edges,
                    weighted=weighted, programs=progs, start=rng.randint(0, 7))
    if kind == "pagerank":
        scale = rng.randint(12, 24)
        fp64 = rng.random() < 0.4
        return dict(kind=kind, graph=rng.choice(["rmat", "rmat", "uniform"]), shuffled=shuffled, scale=scale,
                    vpt=_vpt(rng, scale), edges=_log(rng, 4 << scale, (8 if fp64 and scale > 22 else 16) << scale),
                    fp64=fp64)
    if kind == "batch":
        lo = rng.randint(12, 16)
        return dict(kind=kind, lo=lo, hi=lo + rng.randint(1, min(7, 20 - lo)), factor=rng.randint(6, 16))
    if kind == "adjoint":
        scale = rng.randint(13, 20)
        return dict(kind=kind, graph="rmat", shuffled=shuffled, scale=scale, vpt=_vpt(rng, scale),
                    edges=_log(rng, 4 << scale, 16 << scale))
    scale = rng.randint(14, 22)
    return dict(kind="ingest", scale=scale, vpt=_vpt(rng, scale), edges=_log(rng, 50000, 50000000),
                chunks=rng.randint(1, 5), weighted=rng.random() < 0.6)


# ---- inputs ----------------------------------------------------------------------------


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _rmat(scale, m, g):
    """m RMAT edges with the graph500 quadrant probabilities, as int32 CUDA tensors."""
    src = torch.empty(m, dtype=torch.int32, device="cuda")
    tgt = torch.empty_like(src)
    for lo in range(0, m, 1 << 25):
        cnt = min(1 << 25, m - lo)
        s = torch.zeros(cnt, dtype=torch.int32, device="cuda")
        t = torch.zeros_like(s)
        for _ in range(scale):
            r = torch.rand(cnt, generator=g, device="cuda")
            down = r >= 0.76
            right = torch.where(down, r >= 0.95, r >= 0.57)
            s.mul_(2).add_(down)
            t.mul_(2).add_(right)
        src[lo:lo + cnt] = s
        tgt[lo:lo + cnt] = t
    return src, tgt


def _lattice(scale, g):
    """Both directions of every link of a 2^ceil(scale/2) x 2^floor(scale/2) grid, a tenth missing."""
    w, h = 1 << ((scale + 1) // 2), 1 << (scale // 2)
    v = torch.arange(w * h, device="cuda", dtype=torch.int32)
    right, down = v[(v % w) < w - 1], v[: w * (h - 1)]
    a, b = torch.cat([right, down]), torch.cat([right + 1, down + w])
    keep = torch.rand(len(a), generator=g, device="cuda") >= 0.1
    a, b = a[keep], b[keep]
    return torch.cat([a, b]).contiguous(), torch.cat([b, a]).contiguous()


def _graph(case, m, g):
    n = 1 << case["scale"]
    if case["graph"] == "lattice":
        s, t = _lattice(case["scale"], g)
    elif case["graph"] == "uniform":
        s = torch.randint(0, n, (m,), generator=g, device="cuda", dtype=torch.int32)
        t = torch.randint(0, n, (m,), generator=g, device="cuda", dtype=torch.int32)
    else:
        s, t = _rmat(case["scale"], m, g)
    if case["shuffled"]:
        p = torch.randperm(n, generator=g, device="cuda", dtype=torch.int32)
        for x in (s, t):
            for lo in range(0, len(x), 1 << 26):
                x[lo:lo + (1 << 26)] = p[x[lo:lo + (1 << 26)].long()]
    return s, t


def _weights(m, g):
    return torch.randint(1, 256, (m,), generator=g, device="cuda", dtype=torch.int32)


def _float_weights(m, g):
    return 0.1 + 0.9 * torch.rand(m, generator=g, device="cuda")


def _simple(case, g):
    """`edges` distinct edges of the case's graph in random order, so that every seed has as many weights."""
    n, m = 1 << case["scale"], case["edges"]
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    while len(keys) < m:
        s, t = _graph(case, 2 * m, g)
        keys = torch.unique(torch.cat([keys, s.long() * n + t.long()]))
    keys = keys[torch.randperm(len(keys), generator=g, device="cuda")[:m]]
    return (keys // n).to(torch.int32), (keys % n).to(torch.int32)


def _batch_scales(case):
    return range(case["lo"], case["hi"] + 1)


def _batch_inputs(case, seed):
    """Per snapshot: scale, edges at first, edges of the update, (src, tgt, weight)."""
    out = []
    for scale in _batch_scales(case):
        g = _gen(seed, scale)
        m = case["factor"] << scale
        b = m // 20
        out.append((scale, m, b, (*_rmat(scale, m + b, g), _weights(m + b, g))))
    return out


_PROGRAMS = {
    "bfs": lambda e, start, it: cg.BFS(e, start_vertex=start, max_iterations=it),
    "cc": lambda e, start, it: cg.CC(e, max_iterations=it),
    "sssp": lambda e, start, it: cg.SSSP(e, start_vertex=start, max_iterations=it),
    "sswp": lambda e, start, it: cg.SSWP(e, start_vertex=start, max_iterations=it),
}


def _programs(case, eng, s, max_iterations=100):
    """The case's programs. They start at a vertex that has edges: low ids are hubs in a graph
    whose ids carry the order, elsewhere the source of one of the first edges is taken."""
    start = case.get("start", 0)
    if case["shuffled"] or case["graph"] != "rmat":
        start = int(s[start])
    return [_PROGRAMS[p](eng, start, max_iterations) for p in case["programs"].split(",")]


def _on_device(progs):
    out = []
    for p in progs:
        dtype = torch.float32 if p.result_dtype == np.float32 else torch.int32
        out.append(p.result(out=torch.empty(p.engine.n, dtype=dtype, device="cuda")))
    return out


def _fill(eng, s, t, w):
    """Inserts and compacts a standing graph in chunks."""
    step = 1 << 27
    for lo in range(0, len(s), step):
        eng.insert_edges(s[lo:lo + step], t[lo:lo + step], w[lo:lo + step] if w is not None else None)
        eng.do_global_compaction()


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    st = {"case": case}
    if kind == "stream":
        m = case["batch"] * case["batches"]
        s, t = _graph(case, m, g)
        w = _weights(m, g) if case["weighted"] else None
        torch.cuda.synchronize()
        eng = cg.Engine(1 << case["scale"], case["vpt"], weight_type=cg.WEIGHT_U32 if case["weighted"] else cg.UNWEIGHTED)
        st.update(eng=eng, progs=_programs(case, eng, s), s=s, t=t, w=w)
        # a long-lived context: its buffers have grown and its kernel shapes are tuned
        _stream(st)
        eng.autotune()
    elif kind == "prdelta":
        s, t = _graph(case, case["batch"] * case["batches"], g)
        eng = cg.Engine(1 << case["scale"], case["vpt"])
        prog = cg.PageRankDelta(eng, delta=0.0, max_iterations=1000, tolerance=1e-7)
        st.update(eng=eng, prog=prog, keep=(s.cpu().pin_memory(), t.cpu().pin_memory()))
        st["s"], st["t"] = (x.numpy().view(np.uint32) for x in st["keep"])
    elif kind == "window":
        n, m = 1 << case["scale"], case["edges"]
        s, t = _graph(case, m + case["batch"], g)
        w = _weights(m + case["batch"], g) if case["weighted"] else None
        # the window's edges: distinct, and none of them stands already
        keys = s.long() * n + t.long()
        base = torch.unique(keys[:m])
        new = torch.unique(keys[m:])
        new = new[~torch.isin(new, base)]
        nw = w[m:m + len(new)] if w is not None else None
        torch.cuda.synchronize()
        eng = cg.Engine(n, case["vpt"], weight_type=cg.WEIGHT_U32 if case["weighted"] else cg.UNWEIGHTED)
        _fill(eng, s[:m], t[:m], w[:m] if w is not None else None)
        host = lambda x: None if x is None else x.to(torch.int32).cpu().numpy().view(np.uint32)  # noqa: E731
        st.update(eng=eng, progs=_programs(case, eng, s), s=host(new // n), t=host(new % n), w=host(nw))
        eng.run_many(st["progs"])
    elif kind in ("traverse", "pagerank"):
        s, t = _graph(case, case["edges"], g)
        weighted = case.get("weighted", False)
        w = _weights(len(s), g) if weighted else None
        torch.cuda.synchronize()
        eng = cg.Engine(1 << case["scale"], case["vpt"], weight_type=cg.WEIGHT_U32 if weighted else cg.UNWEIGHTED)
        _fill(eng, s, t, w)
        if kind == "traverse":
            progs = _programs(case, eng, s, 100 if case["graph"] != "lattice" else 100000)
        else:
            progs = [cg.PageRank(eng, max_iterations=1000, tolerance=1e-9, kahan=not case["fp64"])]
        st.update(eng=eng, progs=progs)
    elif kind == "batch":
        snaps = []
        inputs = _batch_inputs(case, seed)
        torch.cuda.synchronize()
        for scale, m, b, edges in inputs:
            e = cg.Engine(1 << scale, min(65536, 1 << (scale - 2)), weight_type=cg.WEIGHT_U32)
            progs = [cg.BFS(e, start_vertex=0), cg.BFS(e, start_vertex=1), cg.CC(e), cg.CC(e),
                     cg.SSSP(e, start_vertex=0), cg.SSSP(e, start_vertex=1),
                     cg.PageRank(e, tolerance=1e-8), cg.PageRank(e, tolerance=1e-8)]
            snaps.append((e, m, b, edges, progs))
        st.update(snaps=snaps)
    elif kind == "adjoint":
        s, t = _simple(case, g)
        w = _float_weights(len(s), g)
        c = torch.randn(1 << case["scale"], generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
        torch.cuda.synchronize()
        eng = cg.Engine(1 << case["scale"], case["vpt"], weight_type=cg.WEIGHT_F32)
        eng.insert_edges(s, t, w.view(torch.int32))
        eng.do_global_compaction()
        st.update(eng=eng, c=c, prog=cg.WeightedPageRank(eng, max_iterations=1000, tolerance=1e-8))
    else:
        eng = cg.Engine(1 << case["scale"], case["vpt"], weight_type=cg.WEIGHT_U32 if case["weighted"] else cg.UNWEIGHTED)
        size = -(-case["edges"] // case["chunks"])
        bufs = [torch.empty(size, dtype=torch.int32, device="cuda") for _ in range(3 if case["weighted"] else 2)]
        st.update(eng=eng, bfs=cg.BFS(eng, start_vertex=0), bufs=bufs, size=size, seed=int(seed) % 100003 + 1)
    return st


# ---- one pass --------------------------------------------------------------------------


def _stream(st):
    """The whole stream on a cleared context: batch k's programs run while batch k + 1 is
    inserted and merged."""
    case, eng, progs = st["case"], st["eng"], st["progs"]
    s, t, w = st["s"], st["t"], st["w"]
    b = case["batch"]
    eng.clear()
    rounds = []
    for k in range(case["batches"]):
        lo, hi = k * b, (k + 1) * b
        eng.insert_edges(s[lo:hi], t[lo:hi], w[lo:hi] if w is not None else None)
        eng.do_global_compaction()
        if k:
            rounds += eng.run_many_wait()
        eng.run_many_async(progs)
    rounds += eng.run_many_wait()
    return [[x["iterations"], x["count_edges"]] for x in rounds]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "stream":
        counts = np.array(_stream(st), np.int64)
        return {"values": _on_device(st["progs"]), "counts": counts}
    if kind == "prdelta":
        eng, prog, b = st["eng"], st["prog"], case["batch"]
        eng.clear()
        out = []
        for k in range(case["batches"]):
            eng.insert_edges(st["s"][k * b:(k + 1) * b], st["t"][k * b:(k + 1) * b])
            prog.execute_algorithm()
            out.append(prog.result())
        return {"ranks": out}
    if kind == "window":
        eng, progs = st["eng"], st["progs"]
        eng.insert_edges(st["s"], st["t"], st["w"])
        eng.run_many(progs)
        new = _on_device(progs)
        deleted = eng.delete_edges(st["s"], st["t"])
        eng.run_many(progs)
        return {"inserted": new, "expired": _on_device(progs), "deleted": deleted}
    if kind == "traverse":
        eng, progs = st["eng"], st["progs"]
        for p in progs:
            p.init_algorithm()
        if len(progs) == 1:
            stats = [progs[0].execute_algorithm()]
        else:
            stats = eng.run_many(progs)
        return {"values": _on_device(progs), "rounds": [x["iterations"] for x in stats]}
    if kind == "pagerank":
        prog = st["progs"][0]
        prog.init_algorithm()
        prog.execute_algorithm()
        return {"ranks": prog.result64() if case["fp64"] else _on_device([prog])[0]}
    if kind == "batch":
        progs = [p for _, _, _, _, ps in st["snaps"] for p in ps]
        for part in (0, 1):
            for e, m, b, (s, t, w), _ in st["snaps"]:
                if part == 0:
                    e.clear()
                lo, hi = (0, m) if part == 0 else (m, m + b)
                e.insert_edges(s[lo:hi], t[lo:hi], w[lo:hi])
                e.do_global_compaction()
            cg.run_batch(progs)
        return {"values": _on_device(progs)}
    if kind == "adjoint":
        prog = st["prog"]
        prog.init_algorithm()
        prog.execute_algorithm()
        gw, gt, _ = prog.adjoint(st["c"])
        return {"ranks": prog.result(), "weights": gw, "teleport": gt}
    eng = st["eng"]
    eng.clear()
    for k in range(case["chunks"]):
        lo = k * st["size"]
        cnt = min(st["size"], case["edges"] - lo)
        bufs = [x[:cnt] for x in st["bufs"]]
        more = dict(weight_seed=st["seed"] + 1000, wmin=1, wmax=255) if case["weighted"] else {}
        eng.generate_rmat(lo, cnt, case["scale"], seed=st["seed"], out=tuple(bufs), **more)
        eng.insert_edges(*bufs)
        eng.do_global_compaction()
    bfs = st["bfs"]
    bfs.execute_algorithm()
    edges, pending = eng.count_edges()
    out_degree, in_degree = eng.degrees()
    return {"levels": _on_device([bfs])[0], "out_degree": out_degree.view(np.int32),
            "in_degree": in_degree.view(np.int32), "edges": [edges, pending]}


# ---- what a pass cannot do without ------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "batch":
        byts = flops = 0.0
        for scale in _batch_scales(case):
            m, n = case["factor"] << scale, 1 << scale
            # loaded, stored, read by eight jobs, updated; ranks iterated
            byts += m * (12 + 8) + m * (4 * 4 + 2 * 8) + 2 * PAGERANK_ROUNDS * m * 8.0 + 8 * n * 4
            flops += m * 8.0 + 2 * PAGERANK_ROUNDS * m * 2.0
        return {"bytes": byts, "flops": flops}
    n, wb = 1 << case["scale"], 4 if case.get("weighted") else 0
    if kind == "stream":
        m, p = case["batch"] * case["batches"], len(case["programs"].split(","))
        return {"bytes": m * (8.0 + wb) + m * (4.0 + wb) * (1 + p) + 4.0 * n * p, "flops": 2.0 * m * p}
    if kind == "prdelta":
        b, k = case["batch"], case["batches"]
        edges = b * k * (k + 1) / 2.0
        return {"bytes": PRDELTA_ROUNDS * edges * 8.0 + b * k * 12.0 + 4.0 * n * k, "flops": PRDELTA_ROUNDS * edges * 2.0}
    if kind == "window":
        p = len(case["programs"].split(","))
        # new edges in and out, one rewrite of the store for each, the programs' answers twice
        return {"bytes": 2.0 * case["edges"] * (8 + 2 * wb) + case["batch"] * (16.0 + wb) + 8.0 * n * p,
                "flops": 2.0 * case["edges"] * p}
    m = case["edges"] or 4 * n
    if kind == "traverse":
        p = case["programs"].split(",")
        byts = sum(m * (8.0 if x in ("sssp", "sswp") else 4.0) + 4.0 * n for x in p)
        return {"bytes": byts, "flops": 2.0 * m * len(p)}
    if kind == "pagerank":
        v = 8.0 if case["fp64"] else 4.0
        return {"bytes": PAGERANK_ROUNDS * (m * (4.0 + v) + 3 * v * n), "flops": PAGERANK_ROUNDS * 2.0 * m}
    if kind == "adjoint":
        r = FORWARD_ROUNDS + ADJOINT_ROUNDS
        return {"bytes": r * (m * 12.0 + 12.0 * n) + 4.0 * m + 16.0 * n, "flops": r * 3.0 * m}
    # ingest: generated, read, stored, read once by the traversal; two hashes of the generator per level
    return {"bytes": m * (2 * (8.0 + wb) + 2 * (4.0 + wb)) + 12.0 * n, "flops": 12.0 * m * case["scale"]}


# ---- the same in 64 bits ----------------------------------------------------------------


def _distinct(s, t, n, w=None):
    """Distinct (src, tgt), sorted; the least weight of each where weights are given."""
    keys = torch.empty(len(s), dtype=torch.int64, device="cuda")
    for lo in range(0, len(s), 1 << 26):
        keys[lo:lo + (1 << 26)] = s[lo:lo + (1 << 26)].long() * n + t[lo:lo + (1 << 26)].long()
    if w is None:
        return torch.unique(keys), None
    k, inv = torch.unique(keys, return_inverse=True)
    ww = torch.full((len(k),), float("inf"), dtype=torch.float64, device="cuda")
    ww.scatter_reduce_(0, inv, w.double(), "amin")
    return k, ww


def _matrix(rows, cols, vals, n):
    """CSR of the given entries; `rows` need not be sorted."""
    o = torch.argsort(rows.long() * n + cols.long())
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return torch.sparse_csr_tensor(ptr, cols[o], vals[o], size=(n, n))


def _pagerank64(keys, n, tol=1e-15):
    u, v = keys // n, keys % n
    d = torch.bincount(u, minlength=n).double()
    p = _matrix(v, u, 1.0 / d[u], n)
    del u, v
    r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    hanging = d == 0
    for _ in range(300):
        new = (1 - ALPHA) / n + ALPHA * (p @ r + r[hanging].sum() / n)
        off = float((new - r).abs().sum())
        r = new
        if off < tol:
            break
    return r


def exact(case, seed):
    kind = case["kind"]
    if kind in ("stream", "window", "traverse", "ingest"):
        return None  # whole numbers
    if kind == "batch":
        out = []
        for scale, m, b, (s, t, w) in _batch_inputs(case, seed):
            n = 1 << scale
            r = _pagerank64(_distinct(s, t, n)[0], n)
            out += [None] * 6 + [r, r]
        return {"values": out}
    g = _gen(seed)
    n = 1 << case["scale"]
    if kind == "prdelta":
        b = case["batch"]
        s, t = _graph(case, b * case["batches"], g)
        out = []
        r = torch.ones(n, dtype=torch.float64, device="cuda")
        for k in range(1, case["batches"] + 1):
            keys = _distinct(s[:k * b], t[:k * b], n)[0]
            d = torch.bincount(s[:k * b].long(), minlength=n).double()  # every copy counts
            u, v = keys // n, keys % n
            p = _matrix(v, u, 1.0 / d[u], n)
            for _ in range(400):
                new = (1 - ALPHA) + ALPHA * (p @ r)
                off = float((new - r).abs().sum() / new.sum())
                r = new
                if off < 1e-15:
                    break
            out.append(r)
        return {"ranks": out}
    if kind == "pagerank":
        s, t = _graph(case, case["edges"], g)
        keys = _distinct(s, t, n)[0]
        del s, t
        return {"ranks": _pagerank64(keys, n)}
    # adjoint: r = (1 - a) t + a (P r + D t), t uniform; lambda = c + a (P^T lambda + a_u (t . lambda))
    s, t = _simple(case, g)
    w = _float_weights(len(s), g)
    c = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    keys, ww = _distinct(s, t, n, w)
    u, v = keys // n, keys % n
    total = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, u, ww)
    vals = ww / total[u]
    p, pt = _matrix(v, u, vals, n), _matrix(u, v, vals, n)
    hanging = total == 0
    r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    for _ in range(300):
        d = r[hanging].sum()
        new = (1 - ALPHA) / n + ALPHA * (p @ r + d / n)
        off = float((new - r).abs().sum())
        r = new
        if off < 1e-15:
            break
    lam = c.clone()
    for _ in range(400):
        q = pt @ lam
        new = c + ALPHA * (q + hanging.double() * lam.mean())
        off = float((new - lam).abs().sum() / c.abs().sum())
        lam = new
        if off < 1e-15:
            break
    q = pt @ lam
    gw = ALPHA * r[u] / total[u] * (lam[v] - q[u])
    # in the order of the store: tile by tile, then by source and target
    vpt = case["vpt"]
    tiles = (u // vpt) * (n // vpt) + v // vpt
    o = torch.argsort((tiles * vpt + u % vpt) * vpt + v % vpt)
    gt = ((1 - ALPHA) + ALPHA * r[hanging].sum()) * lam
    return {"ranks": r, "weights": gw[o], "teleport": gt}
