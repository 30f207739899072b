"""Benchmark: pattern counts per second on RMAT scale 22 (the reference's
eight single-pattern workload), on N GPUs of one node.

One step = one pass of the counting path over the workload: the graph's
loader passes (degree orientation, triangle supports) plus the eight counts,
each result read back to the host.

  value   inputs resident in HBM (a device copy of the raw CSR) when the timed
          region starts; CUDA events on the context stream
  e2e     the same step through the C ABI from pinned host buffers, the CSR
          upload and the result read-back inside the timed region
  --impl reference
          the reference's own counting kernels on the same GPU and graph (its
          src/fringeCount.cu compiled for sm_103a, run by oracle/ref_runner,
          timed as its `runtime:` line), one process per pattern and no
          product code loaded; passes repeat within --ref-budget seconds
  cpu_baseline
          the oracle's CPU restatement of the reference's per-match formulas on
          the host cores, on a hashed sample of each pattern's work items,
          scaled to the whole workload (the reference has no CPU path)

Untimed, after the measurement, the line also carries the exact 128-bit count
of each pattern (fsgc_count_exact) beside the reference-compatible u64 one, and
whether the u64 arithmetic wrapped (--no-exact skips it).

Other workloads (one JSON line each, not the default):
  --workload mixed    batching on one graph: 64 seeded mixed patterns counted in
                      shared passes from a captured CUDA graph, against one
                      fsgc_count per pattern
  --workload packed   batching across graphs: seeded Chung-Lu member graphs in
                      one packed CSR, one count per pattern, against one
                      fsgc_count per (graph, pattern)
  --workload serve    the serving loop: resident RMAT graphs, Poisson arrivals
                      of (graph, pattern) queries, p50/p99 latency, then the
                      same queries as a burst with and without batching

Multi-GPU: replicas only (each rank counts the whole workload on its own
GPU); value = all ranks' patterns / the slowest rank's time.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "fringe-sgc_gb300"))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

WORKLOAD = {
    "wedge_1_on_centre": (4, [(0, 1), (0, 2), (0, 3)]),
    "wedge_2_on_centre": (5, [(0, 1), (0, 2), (0, 3), (0, 4)]),
    "wedge_4_on_centre": (7, [(0, 1), (0, 2), (0, 3), (0, 4), (0, 5), (0, 6)]),
    "wedge_1_on_each_end": (5, [(0, 1), (0, 2), (1, 3), (2, 4)]),
    "triangle_3_on_one": (6, [(0, 1), (1, 2), (0, 2), (0, 3), (0, 4), (0, 5)]),
    "4cycle_opposite": (6, [(0, 1), (1, 2), (2, 3), (3, 0), (0, 4), (2, 5)]),
    "4clique_3_distinct": (7, [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3), (0, 4), (1, 5), (2, 6)]),
    "edge_5_5": (12, [(0, 1)] + [(0, i) for i in range(2, 7)] + [(1, i) for i in range(7, 12)]),
}
# Core shapes of the mixed-pattern workloads (batching and serving): each
# drawn pattern is one of these cores plus 0-12 fringe vertices, each fringe
# adjacent to a uniformly random nonempty subset of the core vertices.
CORE_SHAPES = {
    "edge": (2, [(0, 1)]),
    "wedge": (3, [(0, 1), (0, 2)]),
    "triangle": (3, [(0, 1), (1, 2), (0, 2)]),
    "4path": (4, [(0, 1), (1, 2), (2, 3)]),
    "4cycle": (4, [(0, 1), (1, 2), (2, 3), (3, 0)]),
    "diamond": (4, [(0, 1), (1, 2), (2, 3), (3, 0), (0, 2)]),
    "4clique": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]),
    "5cycle": (5, [(0, 1), (1, 2), (2, 3), (3, 4), (4, 0)]),
}
RMAT = dict(scale=22, edge_factor=16, a=0.57, b=0.19, c=0.19, seed=20251203)
METRIC = "pattern counts/s (RMAT-22, 8 single patterns)"
UNIT = "patterns/s"


def load_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi samples during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except (FileNotFoundError, OSError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.lines:
            return None
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm)}


def workload_graph(scale=None):
    import fsgc
    t = time.time()
    g = fsgc.gen_rmat(scale or RMAT["scale"], RMAT["edge_factor"], RMAT["a"], RMAT["b"], RMAT["c"], RMAT["seed"])
    return g, time.time() - t


def matching_orders(names=None):
    import fsgc
    return [(name, fsgc.preprocess(n, e)) for name, (n, e) in WORKLOAD.items() if not names or name in names]


def draw_patterns(count, seed, max_fringes=12, max_core=6):
    """Seeded mixed patterns: a core shape, then 0..max_fringes fringe vertices
    each joined to a uniformly random nonempty subset of the core vertices.
    Draws whose decomposition is refused (a core of more than six vertices) or
    whose decomposed core has more than max_core vertices are drawn again.
    Returns [(name, MatchingOrder)].

    max_core=3 keeps the vertex, edge, wedge and triangle cores.  Cores of four
    or more vertices sum, per core match, the reference's fringe-placement
    enumeration (src/fringeCount.cu:408-486), whose cost grows exponentially
    with the number of anchor sets: with five or more anchor sets the oracle
    needs more than 20 s on a 256-vertex RMAT graph, and the match count grows
    by orders of magnitude per RMAT scale."""
    import fsgc
    rng = np.random.default_rng(seed)
    names = list(CORE_SHAPES)
    out = []
    while len(out) < count:
        shape = names[int(rng.integers(len(names)))]
        k, core = CORE_SHAPES[shape]
        nf = int(rng.integers(0, max_fringes + 1))
        edges = list(core)
        for i in range(nf):
            sub = int(rng.integers(1, 1 << k))
            edges += [(j, k + i) for j in range(k) if sub >> j & 1]
        try:
            mo = fsgc.preprocess(k + nf, edges)
        except fsgc.FsgcError:
            continue
        if mo.nodes > max_core:
            continue
        out.append((f"{shape}+{nf}#{len(out)}", mo))
    return out


def wedge_bytes(g):
    """Algorithmic bytes of the wedge-pair kernel: every centre u lists each
    pair of its neighbours once (4 bytes per neighbour-list entry read)."""
    d = g.degrees().astype(np.float64)
    return 4.0 * float((d * (d - 1) / 2).sum())


def kernel_bytes(name, core, g):
    d = g.degrees().astype(np.float64)
    if core == 1:
        return 4.0 * g.n  # degree array
    if core == 2 and name == "triangle_3_on_one":
        return 12.0 * g.n  # per-vertex triangle counts + degrees
    if core == 2:
        return 12.0 * g.m / 2  # oriented edge endpoints + support
    if core == 3:
        return wedge_bytes(g)
    if core == 4:
        return triangle_bytes(g)
    return None


def triangle_bytes(g, chunk=1 << 24):
    """Entries of the oriented lists that the triangle core reads: every neighbour
    x of a lowest vertex has its list read once per lower vertex beside it, 4
    bytes for each of sum over x of deg(x) * outdeg(x) entries."""
    d = g.degrees().astype(np.int64)
    key = d * g.n + np.arange(g.n)
    total, v = 0.0, 0
    while v < g.n:
        e = max(v + 1, int(np.searchsorted(g.nindex, g.nindex[v] + chunk, side="right")) - 1)
        a, b = int(g.nindex[v]), int(g.nindex[e])
        up = np.concatenate([[0], np.cumsum(key[g.nlist[a:b]] > np.repeat(key[v:e], d[v:e]))])
        at = np.asarray(g.nindex[v:e + 1], dtype=np.int64) - a
        total += float(np.dot((up[at[1:]] - up[at[:-1]]).astype(np.float64), d[v:e].astype(np.float64)))
        v = e
    return 4.0 * total


def edges_per_second(m, per_pattern_ms):
    """The reference harness's throughput figure per pattern: directed CSR
    entries / count seconds (reproduce.py:91)."""
    return {k: (m / (ms / 1000.0) if ms > 0 else None) for k, ms in per_pattern_ms.items()}


def measured_traffic(pattern, g):
    """DRAM bytes (read + write) of one count of `pattern` on this graph, from the
    ncu captures recorded in profiles/dram_traffic.json (null when none is of this
    pattern and graph size)."""
    p = os.path.join(ROOT, "profiles", "dram_traffic.json")
    if not os.path.exists(p):
        return None
    with open(p) as f:
        rec = json.load(f)
    for r in [rec] + rec.get("others", []):
        if (r.get("pattern"), r.get("n"), r.get("m")) == (pattern, g.n, g.m):
            return r.get("dram_bytes")
    return None


def max_over_ranks(values, world):
    """Replicas: the job's time is the slowest rank's (element-wise max over ranks)."""
    if world <= 1:
        return list(values)
    import torch
    import torch.distributed as dist
    # NCCL reduces device tensors only; gloo (CPU tests) host tensors
    device = f"cuda:{torch.cuda.current_device()}" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor(values, dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return [float(x) for x in t.cpu()]


def job_value(patterns_per_rank, steps, world, seconds):
    """Whole-job throughput: every rank counts the whole workload (replicas)."""
    return patterns_per_rank * world * steps / seconds


def apply_tuning(ctx, g):
    """The autotuner's values for this graph (fringe-sgc_gb300/tuning.json,
    written by fringe-sgc_gb300/autotune.py on a GB300), else the defaults.
    Returns what the line reports."""
    import autotune
    key = autotune.graph_key(g.n, g.m, int(g.degrees().max()))
    values = autotune.load(os.path.join(ROOT, "fringe-sgc_gb300", "tuning.json"), key)
    if values:
        ctx.set_tuning(None, **values)
        return {"source": "fringe-sgc_gb300/tuning.json (autotune.py)", "values": values}
    return {"source": "defaults", "values": ctx.get_tuning().as_dict()}


def run_gpu(args, rank, world):
    import fsgc
    dev = int(os.environ.get("LOCAL_RANK", "0"))
    ctx = fsgc.Context(dev)
    g, gen_s = workload_graph(args.scale)
    tuning = apply_tuning(ctx, g)
    mos = matching_orders(args.patterns)
    tasks_of = lambda gid: [(gid, mo) for _, mo in mos]  # noqa: E731
    # raw CSR resident in HBM for the device-resident measurement
    import ctypes as C
    L = fsgc.lib()
    cudart = None
    d_idx = C.c_void_p()
    d_adj = C.c_void_p()
    try:
        import torch
        t_idx = torch.from_numpy(g.nindex).to(f"cuda:{dev}")
        t_adj = torch.from_numpy(g.nlist).to(f"cuda:{dev}")
        torch.cuda.synchronize(dev)
        d_idx, d_adj = t_idx.data_ptr(), t_adj.data_ptr()
    except ImportError:
        raise SystemExit("torch is needed for the device-resident copy of the input")
    # pinned host copy for e2e
    h = g.as_host_csr()
    L.fsgc_host_csr_pin(C.byref(h))

    def step_device():
        gid = ctx.upload_device(g.n, g.m, d_idx, d_adj)
        ctx.prepare(gid)
        res = ctx.count_batch(tasks_of(gid))
        ctx.release(gid)
        return res

    def step_host():
        gid = ctx.upload(g)
        res = ctx.count_batch(tasks_of(gid))
        ctx.release(gid)
        return res

    barrier = (lambda: __import__("torch").distributed.barrier()) if world > 1 else (lambda: None)
    for _ in range(args.warmup):
        ref_res = step_device()
    # timed: device-resident
    launches0 = ctx.launches
    barrier()
    ctx.synchronize()
    per_step = []
    per_task = np.zeros(len(mos))
    prep_ms = []
    with ClockSampler(dev) as clk:
        for _ in range(args.steps):
            ctx.flush_l2()
            ctx.timer_start()
            gid = ctx.upload_device(g.n, g.m, d_idx, d_adj)
            ctx.prepare(gid)
            prep_ms.append(ctx.timer_stop())
            res = ctx.count_batch(tasks_of(gid))
            ctx.release(gid)
            per_task += np.array([r.device_ms for r in res])
            per_step.append(prep_ms[-1] + sum(r.device_ms for r in res))
            for a, b in zip(res, ref_res):
                assert a.count == b.count, "count changed between steps"
    ctx.synchronize()
    barrier()
    launches = ctx.launches - launches0
    t_dev = sum(per_step) / 1000.0
    # e2e through the C ABI from pinned host memory, wall clock
    barrier()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        res_h = step_host()
    t_e2e = time.perf_counter() - t0
    barrier()
    for a, b in zip(res_h, ref_res):
        assert a.count == b.count
    # exact 128-bit counts beside the reference-compatible u64 ones (untimed)
    exact = {}
    if args.exact:
        gid = ctx.upload(g)
        try:
            for (name, mo), r in zip(mos, ref_res):
                x = ctx.count_exact(gid, mo)
                exact[name] = {"exact": "saturated" if x.saturated else str(x.count),
                               "u64_wrapped": x.saturated or x.raw_total != r.raw_total}
        except fsgc.FsgcError as e:  # reported, not fatal: the timed numbers stand
            exact["error"] = str(e)
        ctx.release(gid)
    t_dev, t_e2e = max_over_ranks([t_dev, t_e2e], world)
    out = {
        "per_task_ms": {name: per_task[i] / args.steps for i, (name, _) in enumerate(mos)},
        "prep_ms": statistics.mean(prep_ms),
        "counts": {name: int(r.count) for (name, _), r in zip(mos, ref_res)},
        "exact": exact,
        "cores": {name: int(r.core_type) for (name, _), r in zip(mos, ref_res)},
        "t_dev": t_dev, "t_e2e": t_e2e, "launches": launches, "clocks": clk.summary(), "gen_s": gen_s,
        "tuning": tuning,
        "graph": {"n": g.n, "m": g.m, "max_degree": int(g.degrees().max())},
    }
    return out, g, mos, ctx


def cpu_sample(g, mos, budget_s, threads):
    """Time the oracle (the reference's per-match formulas on the host cores)
    on a hashed sample of each pattern's work items (the reference's worklist
    entries), and extrapolate: t_full = t_scan + (t_sample - t_scan) * stride,
    where t_scan is the cost of a pass that takes no item."""
    import oracle
    per = budget_s / len(mos)
    est, samples = 0.0, {}
    for name, mo in mos:
        b = mo.to_bytes()
        t0 = time.perf_counter()
        oracle.count(g.nindex, g.nlist, b, stride=1 << 30, phase=1 << 29, threads=threads)
        t_scan = time.perf_counter() - t0
        stride = 1 << 24
        while True:
            t0 = time.perf_counter()
            oracle.count(g.nindex, g.nlist, b, stride=stride, phase=stride // 3, threads=threads)
            t = time.perf_counter() - t0
            work = max(t - t_scan, 0.0)
            if work >= per / 2 or stride == 1 or t >= per:
                break
            # aim the next sample at ~per/2 seconds of work
            grow = 16 if work <= 0 else min(16.0, max(2.0, (per / 2) / work))
            stride = max(1, int(stride / grow))
        est += t_scan + work * stride
        samples[name] = stride
    return est, samples


def mixed_graphs(count, nmax, seed):
    """Chung-Lu member graphs of uneven size: n log-uniform in [1000, nmax],
    average degree uniform in [4, 64], exponent uniform in [2.1, 2.8]."""
    import fsgc
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        n = int(round(float(np.exp(rng.uniform(np.log(1000), np.log(nmax))))))
        d, e = float(rng.uniform(4, 64)), float(rng.uniform(2.1, 2.8))
        out.append(fsgc.gen_chung_lu(n, d, e, seed * 1000003 + i))
    return out


def run_packed(args):
    """Batching across graphs: every member graph counted with the same
    patterns, (a) packed -- one count per pattern covering all members -- and
    (b) one fsgc_count per (graph, pattern).  Both wall-clock, results read
    back; every per-(graph, pattern) count must agree."""
    import fsgc
    ctx = fsgc.Context(0)
    t = time.time()
    graphs = mixed_graphs(args.graphs, args.nmax, 20251204)
    gen_s = time.time() - t
    pats = draw_patterns(8, 20251205, max_core=3)
    pid = ctx.upload_packed(graphs)
    ctx.prepare(pid)
    gids = [ctx.upload(g) for g in graphs]
    for gid in gids:
        ctx.prepare(gid)
    nq = len(graphs) * len(pats)
    launches0 = ctx.launches
    for _ in range(args.warmup):
        packed = [ctx.count_packed(pid, mo) for _, mo in pats]
    ctx.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        packed = [ctx.count_packed(pid, mo) for _, mo in pats]
    t_packed = (time.perf_counter() - t0) / args.steps
    launches = (ctx.launches - launches0) // (args.steps + args.warmup)
    single = None
    t0 = time.perf_counter()
    for _ in range(max(1, args.steps // 2)):
        single = [[ctx.count(gid, mo) for gid in gids] for _, mo in pats]
    t_single = (time.perf_counter() - t0) / max(1, args.steps // 2)
    for pi in range(len(pats)):
        for gi in range(len(graphs)):
            a, b = packed[pi][gi], single[pi][gi]
            assert (a.count, a.raw_total, a.flags) == (b.count, b.raw_total, b.flags), (pi, gi)
    line = {"metric": "queries/s, batched across graphs (packed CSR, one count per pattern)",
            "value": nq / t_packed, "unit": "queries/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": t_packed * 1000, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "u64", "data": "synthetic",
            "config": {"workload": f"{len(graphs)} Chung-Lu graphs, n log-uniform [1000, {args.nmax}], avg degree "
                                   "U[4,64], exponent U[2.1,2.8], packed into one CSR; 8 mixed patterns",
                       "n_total": int(sum(g.n for g in graphs)), "m_total": int(sum(g.m for g in graphs)),
                       "patterns": [n for n, _ in pats], "gen_s": round(gen_s, 1)},
            "one_query_per_launch": {"value": nq / t_single, "unit": "queries/s", "ms_per_step": t_single * 1000},
            "batched_over_single": (nq / t_packed) / (nq / t_single),
            "gpu_launches": launches, "exact": "all per-(graph, pattern) counts equal"}
    print(json.dumps(line))
    ctx.close()


def per_match_family(mo):
    """True for the patterns whose kernels evaluate a formula per core match
    with a per-match intersection: general cores (4-6 core vertices) and wedge
    cores whose centre carries fringes (the reference's general_wedge_core,
    src/fringeCount.cu:1513-1650).  Their work grows with the number of
    wedges or core paths, one to two orders of magnitude per two RMAT scales."""
    b = mo.to_bytes()
    nodes = b[0]
    if nodes >= 4:
        return True
    if nodes != 3 or bin(b[9]).count("1") != 1:
        return False
    f = [0] * 8
    for i in range(b[1]):
        f[b[13 + i] & 7] = b[76 + i]
    if b[9] == 2:  # centre is B
        f[1], f[2], f[5], f[6] = f[2], f[1], f[6], f[5]
    return bool(f[7] or f[3] or f[5] or f[1])


def placement_bound(mo):
    """Upper bound on the fringe placements a general core enumerates per core
    match: per anchor set, multisets of its fringes over the regions that
    contain it."""
    from math import comb
    b = mo.to_bytes()
    sets = b[1]
    anch, fcnt = b[13:13 + sets], b[76:76 + sets]
    top = 0
    for a in anch:
        top |= a
    bound = 1
    for a, f in zip(anch, fcnt):
        regions = 1 << (bin(top).count("1") - bin(a).count("1"))
        bound *= comb(regions + f - 1, f)
    return bound


def run_mixed(args):
    """Batching on one graph: `--mixed-patterns` seeded patterns drawn as the
    batching configuration describes (core from edge, wedge, triangle,
    4-path, 4-cycle, diamond, 4-clique, 5-cycle; 0-12 fringes each on a random
    non-empty core subset), all on one RMAT graph.

      batched  fsgc_count_set over the patterns: shared passes per core
               family; the first call runs the launches, the second captures
               them into a CUDA graph, the timed calls replay it
      single   one fsgc_count per pattern (one query per launch)

    Patterns whose kernels evaluate a formula per core match with a
    per-match intersection (general cores, and wedge cores whose centre
    carries fringes: per_match_family) have work that grows by one to two
    orders of magnitude per two RMAT scales, so they run on the RMAT graph of
    scale --general-scale, with the same two modes, cheapest first by their
    fringe-placement bound, within --general-budget seconds of single counts
    (the others within --mixed-budget seconds on the main graph, in the same
    order); the rest are listed, not timed (a general core enumerates every fringe
    placement of every core match, and for drawn patterns with many anchor
    sets that is billions of steps even on a 64-vertex graph).  Every batched
    count equals its single count."""
    import fsgc
    ctx = fsgc.Context(0)
    pats = draw_patterns(args.mixed_patterns, 20251208, max_core=6)
    small = [(n, mo) for n, mo in pats if not per_match_family(mo)]
    general = [(n, mo) for n, mo in pats if per_match_family(mo)]

    def measure(scale, group, budget_s=None):
        t = time.time()
        g = fsgc.gen_rmat(scale, RMAT["edge_factor"], RMAT["a"], RMAT["b"], RMAT["c"], RMAT["seed"])
        gen_s = time.time() - t
        gid = ctx.upload(g)
        ctx.prepare(gid)
        tuning = apply_tuning(ctx, g)
        not_timed = []
        if budget_s is not None:
            # cheapest first by the fringe-placement enumeration bound; what
            # does not fit the budget is listed, not timed
            group = sorted(group, key=lambda p: (p[1].nodes, placement_bound(p[1])))
            kept, t0 = [], time.time()
            for name, mo in group:
                if time.time() - t0 > budget_s:
                    not_timed.append(name)
                    continue
                t1 = time.time()
                ctx.count(gid, mo)
                kept.append((name, mo))
                print(f"mixed: RMAT-{scale} {name} {time.time() - t1:.2f} s", file=sys.stderr, flush=True)
            group = kept
        mos = [mo for _, mo in group]
        single = [ctx.count(gid, mo) for mo in mos]  # also builds every per-graph structure
        ctx.synchronize()
        t0 = time.perf_counter()
        for _ in range(max(1, args.steps // 2)):
            single = [ctx.count(gid, mo) for mo in mos]
        t_single = (time.perf_counter() - t0) / max(1, args.steps // 2)
        for _ in range(max(2, args.warmup)):  # direct, then captured
            batched = ctx.count_set(gid, mos)
        ctx.synchronize()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            batched = ctx.count_set(gid, mos)
        t_batched = (time.perf_counter() - t0) / args.steps
        for (name, _), a, b in zip(group, batched, single):
            assert (a.count, a.raw_total, a.automorphisms, a.core_type) == \
                   (b.count, b.raw_total, b.automorphisms, b.core_type), name
        per = {name: round(r.device_ms, 3) for (name, _), r in zip(group, single)}
        ctx.release(gid)
        return {"scale": scale, "n": g.n, "m_directed": g.m, "patterns": len(mos), "gen_s": round(gen_s, 1),
                "batched_queries_per_s": len(mos) / t_batched, "batched_ms": t_batched * 1000,
                "single_queries_per_s": len(mos) / t_single, "single_ms": t_single * 1000,
                "batched_over_single": t_single / t_batched, "single_per_pattern_ms": per, "tuning": tuning,
                "counts": {name: str(r.count) for (name, _), r in zip(group, single)},
                "not_timed": not_timed}

    launches0 = ctx.launches
    main_part = measure(args.mixed_scale, small, args.mixed_budget)
    gen_part = measure(args.general_scale, general, args.general_budget) if general else None
    line = {"metric": "queries/s, mixed patterns on one graph (batched in shared passes from a captured CUDA graph)",
            "value": main_part["batched_queries_per_s"], "unit": "queries/s", "n_gpus": 1, "steps": args.steps,
            "warmup": max(2, args.warmup), "ms_per_step": main_part["batched_ms"], "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u64", "data": "synthetic",
            "config": {"workload": f"{args.mixed_patterns} seeded mixed patterns (seed 20251208); "
                                   f"{len(small)} on RMAT scale {args.mixed_scale}; the {len(general)} general "
                                   f"cores and fringed-centre wedges on RMAT scale {args.general_scale}",
                       "main": main_part, "general": gen_part},
            "one_query_per_launch": {"value": main_part["single_queries_per_s"], "unit": "queries/s",
                                     "ms_per_step": main_part["single_ms"]},
            "batched_over_single": main_part["batched_over_single"],
            "gpu_launches": ctx.launches - launches0,
            "exact": "every batched count equals the single count of the same pattern"}
    print(json.dumps(line))
    ctx.close()


def run_serve(args):
    """Serving: resident RMAT graphs, Poisson arrivals of (random graph, random
    mixed pattern) queries into fsgc_server_*, p50/p99 latency and queries/s,
    then the same queries as one closed burst with continuous batching and with
    one query per launch (one lane, batches of one).  Every served count is
    compared with a direct count of the same query."""
    import fsgc
    ctx = fsgc.Context(0)
    scales = [int(x) for x in args.serve_scales.split(",")]
    t = time.time()
    graphs = [fsgc.gen_rmat(sc, RMAT["edge_factor"], RMAT["a"], RMAT["b"], RMAT["c"], RMAT["seed"] + sc)
              for sc in scales]
    gen_s = time.time() - t
    gids = [ctx.upload(g) for g in graphs]
    graph_sizes = [(g.n, g.m) for g in graphs]
    del graphs  # the host copies (tens of GB at the larger scales)
    # per-match families (general cores, fringed-centre wedges) are left out:
    # at these scales one such query enumerates 10^12 and more core matches
    pats = [(n, mo) for n, mo in draw_patterns(64, 20251206, max_core=3) if not per_match_family(mo)]
    rng = np.random.default_rng(20251207)
    nq = args.queries
    qs = [(int(rng.integers(len(gids))), int(rng.integers(len(pats)))) for _ in range(nq)]
    gaps = rng.exponential(1.0 / args.rate, nq)
    # pattern divisors and per-graph structures are built once, before serving
    direct = {}
    t = time.time()
    for gi, pi in sorted(set(qs)):
        direct[(gi, pi)] = ctx.count(gids[gi], pats[pi][1])
    print(f"serve: {len(direct)} direct counts in {time.time() - t:.1f} s", file=sys.stderr, flush=True)
    budget = int(args.budget_gb * (1 << 30))

    def serve(lanes, max_batch, arrivals):
        with fsgc.Server(ctx, budget, lanes=lanes, max_batch=max_batch) as srv:
            for gid in gids:
                srv.add_graph(gid)
            tickets = []
            t0 = time.perf_counter()
            at = 0.0
            for k, (gi, pi) in enumerate(qs):
                if arrivals:
                    at += gaps[k]
                    d = t0 + at - time.perf_counter()
                    if d > 0:
                        time.sleep(d)
                tickets.append(srv.submit(gids[gi], pats[pi][1]))
            res = [srv.wait(tk, timeout_s=3600) for tk in tickets]
            st = srv.stats()
            wall = time.perf_counter() - t0
        for (gi, pi), (r, _) in zip(qs, res):
            d = direct[(gi, pi)]
            assert (r.count, r.raw_total) == (d.count, d.raw_total), (gi, pi)
        return {"queries_per_s": st.queries_per_s, "p50_ms": st.p50_ms, "p99_ms": st.p99_ms,
                "rounds": int(st.rounds), "cache_hits": int(st.cache_hits), "wall_s": wall}

    launches0 = ctx.launches
    poisson = serve(args.lanes, 64, True)
    launches = ctx.launches - launches0
    print(f"serve: poisson {poisson}", file=sys.stderr, flush=True)
    burst = single = None
    if args.serve_burst:
        burst = serve(args.lanes, 64, False)
        print(f"serve: burst {burst}", file=sys.stderr, flush=True)
        single = serve(1, 1, False)
    line = {"metric": f"served queries/s at Poisson {args.rate:g}/s offered (p50/p99 latency beside)",
            "value": poisson["queries_per_s"], "unit": "queries/s", "n_gpus": 1, "steps": 1, "warmup": 0,
            "ms_per_step": poisson["wall_s"] * 1000, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "u64", "data": "synthetic",
            "config": {"workload": f"{len(gids)} resident RMAT graphs (scales {scales}, edge factor 16), "
                                   f"{nq} queries, uniform graph x {len(pats)} mixed patterns (of 64 drawn, "
                                   "without general cores and fringed-centre wedges)",
                       "graphs": [{"scale": sc, "n": n, "m_directed": m} for sc, (n, m) in zip(scales, graph_sizes)],
                       "distinct_queries": len(direct),
                       "lanes": args.lanes, "budget_gb": args.budget_gb, "gen_s": round(gen_s, 1)},
            "p50_ms": poisson["p50_ms"], "p99_ms": poisson["p99_ms"], "poisson": poisson,
            "burst_batched": burst, "burst_one_query_per_launch": single,
            "batched_over_single": (burst["queries_per_s"] / max(single["queries_per_s"], 1e-12)) if burst else None,
            "gpu_launches": launches, "exact": "every served count equals the direct count"}
    print(json.dumps(line))
    ctx.close()


def reference_golden(scale):
    """Counts and times of the reference's own kernels on the benchmark graph at
    `scale` (tests/golden/reference_rmat<scale>.json, written on a GB300 by
    tests/golden/make_reference_counts.py), or None."""
    p = os.path.join(ROOT, "tests", "golden", f"reference_rmat{scale}.json")
    if not os.path.exists(p):
        return None
    with open(p) as f:
        return json.load(f)


def run_reference(args, names):
    """The reference arm: the reference's own counting kernels (its
    src/fringeCount.cu compiled for sm_103a, oracle/_ref/fringeCount.cubin)
    driven by oracle/_build/ref_runner, which repeats occurrences()'s host steps
    and times each count as the reference's `runtime:` line does.  One process
    per pattern, as the reference's harness runs fringeCount.  The graph is
    written by oracle/_build/graphgen and the .mo bytes are the reference
    CLI's own; nothing here loads the product library.

    A pass counts every pattern once, shortest first.  Passes repeat, up to
    warmup + steps, while the next pass is expected to end within --ref-budget
    seconds; the first passes are untimed warm-up when more than one pass fits.
    A pattern is started only when its time in the last pass (or, for the first
    pass, in the recorded full run of the reference's kernels for this scale,
    tests/golden/reference_rmat<scale>.json) fits the remaining budget; a
    pattern that cannot run is named with that recorded time and the line's
    value counts it at that time, stated in the line.  At RMAT scale 22 one
    pass takes the reference about 49 minutes (three patterns of 10-19 minutes
    each), more than one arm may run, so the default budget times the five
    short patterns and the 4-clique one live and takes the two wedge-pair
    patterns from the recorded run."""
    import tempfile
    import refrun
    scale = args.scale or RMAT["scale"]
    base = {"metric": METRIC, "unit": UNIT, "impl": "reference", "n_gpus": 1, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u64", "data": "synthetic"}
    if not refrun.available():
        print(json.dumps({"impl": "reference", "unavailable": "the reference's kernels were not compiled "
                          "(oracle/_ref/fringeCount.cubin is built only where the reference sources are)"}))
        return
    golden = reference_golden(scale)
    expect = {k: v["ms"] / 1000.0 for k, v in (golden or {}).get("patterns", {}).items()}
    # shortest first, so that as many patterns as possible are timed live
    names = sorted(names, key=lambda k: expect.get(k, 0.0))
    mos = refrun.workload_matching_orders(names)
    t_start = time.time()
    deadline = t_start + args.ref_budget
    want = args.warmup + args.steps
    passes, skipped = [], {}
    with tempfile.TemporaryDirectory() as tmp:
        egr = os.path.join(tmp, "g.egr")
        refrun.write_rmat_egr(egr, scale, RMAT["edge_factor"], RMAT["a"], RMAT["b"], RMAT["c"], RMAT["seed"])
        gen_s = time.time() - t_start
        n, m = refrun.egr_header(egr)
        paths = dict(zip(names, refrun.write_mo_files(mos, tmp)))
        while len(passes) < want:
            this = {}
            for name in names:
                guess = passes[-1][name]["ms"] / 1000.0 if passes else expect.get(name, 0.0)
                if time.time() + 1.2 * guess + 5.0 > deadline:
                    if passes:
                        break
                    skipped[name] = guess
                    continue
                t0 = time.time()
                r = refrun.run(egr, [paths[name]])[0]
                r["wall_s"] = time.time() - t0
                this[name] = r
                print(f"reference: pass {len(passes)} {name} {r['ms']:.1f} ms", file=sys.stderr, flush=True)
            if len(this) < len(names):
                if not passes:
                    passes.append(this)  # the first, incomplete pass still reports what ran
                break
            passes.append(this)
            if time.time() + sum(r["wall_s"] for r in this.values()) > deadline:
                break
    complete = [p for p in passes if len(p) == len(names)]
    counts = {}
    for p in passes:
        for name, r in p.items():
            counts[name] = {"count": str(r["count"]), "raw": str(r["raw"]), "aut": r["aut"], "core": r["core"]}
    if complete:
        timed = complete[min(args.warmup, len(complete) - 1):]
        step_s = [sum(r["ms"] for r in p.values()) / 1000.0 for p in timed]
        t = statistics.mean(step_s)
        per = {name: statistics.mean(p[name]["ms"] for p in timed) for name in names}
        bound = None
    else:
        timed = []
        ran = passes[0] if passes else {}
        per = {name: r["ms"] for name, r in ran.items()}
        t = (sum(per.values()) / 1000.0) + sum(skipped.values())
        bound = ("upper: " + ", ".join(f"{k} not run (expected {v:.0f} s, from the recorded full run)"
                                       for k, v in skipped.items()) + " and counted at that time")
    value = len(names) / t
    line = dict(base)
    line.update({
        "value": value, "steps": len(timed), "warmup": (len(complete) - len(timed)) if complete else 0,
        "ms_per_step": t * 1000.0,
        "config": {"workload": f"RMAT scale {scale}, edge factor 16, (a,b,c,d)=(.57,.19,.19,.05), "
                               f"{len(names)} single patterns",
                   "n": n, "m_directed": m, "patterns": names,
                   "requested_steps": args.steps, "requested_warmup": args.warmup,
                   "budget_s": args.ref_budget, "graph_gen_s": round(gen_s, 1),
                   "per_pattern_ms": {k: round(v, 3) for k, v in per.items()},
                   "edges_per_s": {k: (round(m / (v / 1000.0), 1) if v > 0 else None) for k, v in per.items()},
                   "counts": counts, "value_bound": bound,
                   "timing": "the reference's runtime: region (src/fringeCount.cu:2317-2321) around occurrences(), "
                             "summed over the patterns; graph file read and upload excluded, as there"},
        "reference_kind": "the reference's own CUDA kernels (src/fringeCount.cu compiled for sm_103a) on this GPU, "
                          "host steps of occurrences() by oracle/ref_runner",
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": None, "kind": "reference",
                         "sample": "the whole workload, no sampling (the reference has no CPU path: its counting "
                                   "path runs as GPU kernels, timed here on the GB300)"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    })
    print(json.dumps(line))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--workload", default="rmat22", choices=["rmat22", "mixed", "packed", "serve"],
                    help="rmat22: the eight-pattern RMAT-22 step (default); mixed: batching many patterns on "
                         "one graph; packed: batching across graphs; serve: the serving loop")
    ap.add_argument("--mixed-patterns", type=int, default=64, help="mixed: patterns drawn")
    ap.add_argument("--mixed-scale", type=int, default=24, help="mixed: RMAT scale for cores of <= 3 vertices")
    ap.add_argument("--general-scale", type=int, default=6,
                    help="mixed: RMAT scale for general cores and fringed-centre wedges")
    ap.add_argument("--general-budget", type=float, default=300.0,
                    help="mixed: seconds of single counts on the general-core graph; patterns beyond it are "
                         "listed, not timed")
    ap.add_argument("--mixed-budget", type=float, default=600.0,
                    help="mixed: seconds of single counts on the main graph; patterns beyond it are listed, "
                         "not timed (the kept patterns are then counted once more singly and max(2, warmup) "
                         "+ steps times as a set, so the run takes up to about (3 + warmup + steps) x this)")
    ap.add_argument("--graphs", type=int, default=256, help="packed: member graphs")
    ap.add_argument("--nmax", type=int, default=50000, help="packed: largest member size")
    ap.add_argument("--serve-scales", default="6,7,8,9,10,11,12,13", help="serve: RMAT scales")
    ap.add_argument("--queries", type=int, default=300, help="serve: queries")
    ap.add_argument("--rate", type=float, default=5.0, help="serve: Poisson arrivals per second")
    ap.add_argument("--lanes", type=int, default=4, help="serve: lanes")
    ap.add_argument("--budget-gb", type=float, default=150.0,
                    help="serve: memory budget (registered graphs and work arenas)")
    ap.add_argument("--serve-burst", type=int, default=1,
                    help="serve: also run the queries as a burst, batched and one per launch")
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="fsgc", choices=["fsgc", "reference"])
    ap.add_argument("--cpu-budget", type=float, default=20.0, help="seconds of CPU-baseline sampling")
    ap.add_argument("--ref-budget", type=float, default=900.0,
                    help="reference arm: seconds within which its passes must end")
    ap.add_argument("--scale", type=int, default=None, help="RMAT scale (profiling runs; default 22)")
    ap.add_argument("--patterns", default=None, help="comma-separated subset of the patterns (profiling runs)")
    ap.add_argument("--no-exact", dest="exact", action="store_false",
                    help="skip the untimed exact 128-bit counts reported beside the u64 ones")
    args = ap.parse_args()
    if args.patterns:
        args.patterns = args.patterns.split(",")
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    threads = os.cpu_count() or 1
    if args.impl == "reference":
        if rank != 0:
            return
        run_reference(args, args.patterns or list(WORKLOAD))
        return
    if args.workload == "mixed":
        if rank == 0:
            run_mixed(args)
        return
    if args.workload == "packed":
        if rank == 0:
            run_packed(args)
        return
    if args.workload == "serve":
        if rank == 0:
            run_serve(args)
        return
    if world > 1:
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
        dist.init_process_group("nccl")
    out, g, mos, ctx = run_gpu(args, rank, world)
    if rank != 0:
        ctx.close()
        if world > 1:
            __import__("torch").distributed.destroy_process_group()
        return
    value = job_value(len(mos), args.steps, world, out["t_dev"])
    e2e = job_value(len(mos), args.steps, world, out["t_e2e"])
    peak, peak_kind = load_peaks()
    # dominant kernel: the task with the largest device time
    dom = max(out["per_task_ms"], key=out["per_task_ms"].get)
    core = out["cores"][dom]
    alg = kernel_bytes(dom, core, g)
    ms = out["per_task_ms"][dom]
    roof = None
    if alg is not None and ms > 0:
        ach = alg / (ms / 1000.0) / 1e9
        roof = {"bound": "hbm", "achieved": round(ach, 1), "peak": peak, "unit": "GB/s",
                "frac": round(ach / peak, 4), "traffic": measured_traffic(dom, g), "kernel": dom,
                "kernel_ms": round(ms, 3), "algorithmic_bytes": alg, "peak_kind": peak_kind}
    cpu = None
    if world == 1 and args.cpu_budget > 0:
        est, samples = cpu_sample(g, mos, args.cpu_budget, os.cpu_count() or 1)
        cpu = {"value": len(mos) / est, "unit": UNIT, "cores": os.cpu_count(), "kind": "port",
               "sample": "oracle on a hashed 1/stride of each pattern's worklist items, strides " +
                         json.dumps(samples) + "; t_scan + (t - t_scan) x stride"}
    h2d = 8 * (g.n + 1) + 4 * g.m
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": out["t_dev"] * 1000 / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u64", "data": "synthetic",
        "config": {"workload": "RMAT scale 22, edge factor 16, (a,b,c,d)=(.57,.19,.19,.05), 8 single patterns",
                   "n": g.n, "m_directed": g.m, "max_degree": out["graph"]["max_degree"],
                   "patterns": list(WORKLOAD), "parallelism": f"replicas x{world}",
                   "l2": "inputs (0.5 GB CSR) larger than L2, and L2 flushed before every timed step",
                   "divisor": "each pattern's divisor (the pattern counted in itself, on its own graph of 4-12 "
                              "vertices) is computed at the first count and cached, so the timed steps leave it "
                              "out; the reference's runtime: line includes it",
                   "prep_ms": round(out["prep_ms"], 3),
                   "per_pattern_ms": {k: round(v, 3) for k, v in out["per_task_ms"].items()},
                   "edges_per_s": {k: (round(v, 1) if v is not None else None)
                                   for k, v in edges_per_second(g.m, out["per_task_ms"]).items()},
                   "counts": out["counts"], "exact_counts": out["exact"],
                   "tuning": out.get("tuning")},
        "roofline": roof,
        "cpu_baseline": cpu,
        "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": 8 * len(mos)},
        "gpu_launches": out["launches"],
        "clocks": out["clocks"],
    }
    print(json.dumps(line))
    ctx.close()
    if world > 1:
        __import__("torch").distributed.destroy_process_group()


if __name__ == "__main__":
    main()
