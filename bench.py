"""Benchmark: exact-depth BFS on the R-MAT scale-22 power-law graph, 1 B200.

Workload (one step): BFS from 64 sources picked as gbench does (largest
component, degree > 0, seed 1; src/bench/main.cpp:155-169) on the R-MAT graph
of 2^22 vertices and 8.5 * 2^22 drawn edges (seed 22; a=.57 b=.19 c=.19),
symmetrised, duplicates and self-loops removed, ids permuted by reorder
"random" seed 1: 4,194,304 vertices, 69,238,210 directed int32 edges
(synthetic stand-in for soc-LiveJournal1).  Each BFS runs as one persistent
cooperative launch with the per-level selector that is faster on the first 16
sources after per-selector autotuning: the learned MLP, or the alpha/beta rule,
which judges it (untimed).  The handle keeps its adjacency lists hub-first on
the device (--adjacency natural keeps the caller's order; depths are the same).  GTEPS = sum over sources of the edges of the
source's component / time (src/bench/main.cpp:329-370).

  value       device-resident: graph in HBM, dist kept on the device, CUDA
              events on the library's stream around one gb_bfs_run_many call
              (the 64 traversals back to back, no host round trip between).
  e2e         the same call returning every source's 16.8 MB uint32 depth
              array to one pinned host buffer inside the timed region (over
              PCIe as 4 bits per depth; each source's copy and host widening
              overlap the next traversals).  compare.e2e_distinct_buffers_gteps:
              the same with a separate host array per source (1 GB per step).
  roofline    persistent kernel, HBM bound: graph-pass bytes 4(n+1)+4m+4n per
              traversal / mean launch time, against the measured copy peak.
  cpu_baseline the reference's own cpu_do (oracle/_ref, all host cores) on a
              bounded sample of the same sources.

python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
Multi-GPU (torchrun): replicas -- every rank runs the full 64-source step on
its own GPU; value = all ranks' edges / max rank time.
"""
from __future__ import annotations

import argparse
import hashlib
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "BFS GTEPS (exact); PR ms/iter & ms-to-tol 1e-6; learned vs rule-based, 1 B200"
WORKLOAD = "rmat22_bfs64"
SCALE, EDGES_DRAWN, GEN_SEED, PERM_SEED, NSRC = 22, 35651584, 22, 1, 64


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.FIELDS,
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = max(mx, float(f[2]))
            except ValueError:
                continue
            for nm, val in zip(names, f[5:9]):
                if val.lower() in ("active", "1"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx or None,
                "reasons": sorted(reasons), "samples": len(sm)}


def build_graph(G, scale=SCALE, nsrc=NSRC, gpu_prep=True):
    """The benchmark graph and its sources.  gpu_prep permutes and picks sources
    with the library's GPU preparation (identical results); the reference arm
    passes False so that its set-up runs on the host only."""
    t = time.time()
    edges = EDGES_DRAWN if scale == SCALE else int(8.5 * (1 << scale))
    g = G.gen.rmat(scale, edges=edges, directed=False, seed=GEN_SEED)
    perm = G.random_perm(g.n, PERM_SEED)
    g = G.permute_gpu(g, perm) if gpu_prep else G.permute(g, perm)
    srcs = G.pick_sources_gpu(g, nsrc, 1) if gpu_prep else G.pick_sources(g, nsrc, 1)
    log(f"graph n={g.n} m={g.m} built in {time.time() - t:.1f}s")
    return g, srcs


def depth_wire_bytes(n, levels):
    """Bytes per depth on the PCIe wire: the library packs depths to 4 bits,
    1 or 2 bytes when the level count allows."""
    if levels < 15:
        return 0.5
    if levels < 255:
        return 1
    if levels < 65535:
        return 2
    return 4


def component_edges(g, dist):
    deg = np.diff(g.row_ptr.astype(np.int64))
    return int(deg[dist != 0xFFFFFFFF].sum()) // 2


def check_depths(g, dist, src):
    """Size-independent validity of a BFS depth array (Graph500 rules)."""
    if dist[src] != 0:
        return False
    u = np.repeat(np.arange(g.n, dtype=np.int64), np.diff(g.row_ptr.astype(np.int64)))
    v = g.col_idx.astype(np.int64)
    du, dv = dist[u].astype(np.int64), dist[v].astype(np.int64)
    unr = 0xFFFFFFFF
    if np.any((du == unr) != (dv == unr)):
        return False
    both = du != unr
    if np.any(np.abs(du[both] - dv[both]) > 1):
        return False
    reached = np.flatnonzero(dist != unr)
    has_parent = np.zeros(g.n, bool)
    m = both & (dv == du - 1)
    has_parent[u[m]] = True
    has_parent[src] = True
    return bool(has_parent[reached].all())


def _oracle():
    """The oracle package (test infrastructure): the reference's own CPU code
    built from its sources (oracle/_ref) and the C restatement.  bench.py
    uses it only as the checker, as the timed CPU baseline and in the
    reference arm -- never on the measured path."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle_py as O
    return O


def depth_hash(d) -> bytes:
    return hashlib.blake2b(np.ascontiguousarray(d).view(np.uint8), digest_size=16).digest()


class ReferenceBfs:
    """The reference's cpu_do (src/cpu/bfs_cpu.cpp:227-283; alpha 15, beta 18,
    all host threads) on a host copy of the graph, from oracle/_ref; the
    oracle's one-thread restatement when the reference build is absent."""

    def __init__(self, n, m, flags, row_ptr, col_idx, ref_graph=None):
        O = _oracle()
        self.deg = np.diff(row_ptr.astype(np.int64))
        if ref_graph is not None or O.ref() is not None:
            self.rg = ref_graph if ref_graph is not None else O.RefGraph.of(
                O.HostGraph(n, m, flags, row_ptr, col_idx))
            self.cores = int(O.ref().gref_max_threads())
            self.kind = "reference"
            self._run = lambda s: self.rg.bfs_do(int(s), 15.0, 18.0, threads=0, trace=False)[0]
        else:
            hg = O.HostGraph(n, m, flags, row_ptr, col_idx)
            self.cores, self.kind = 1, "port"
            self._run = lambda s: O.bfs_do(hg, int(s))[0]

    def run(self, s):
        """(depths, seconds)"""
        t0 = time.perf_counter()
        d = self._run(s)
        return d, time.perf_counter() - t0

    def comp_edges(self, d) -> int:
        return int(self.deg[d != 0xFFFFFFFF].sum()) // 2


def check_against_reference(g, sources, own, hashes, ref=None, timed=64):
    """Every source's GPU depths against the reference's cpu_do, bit for bit.
    own: {source index: GPU depth array} compared element-wise; hashes: {source
    index: 16-byte digest of the GPU depths} for depths held elsewhere (other
    ranks).  Returns (ok, first mismatch, per-source component edges from the
    REFERENCE depths -- the TEPS denominators of src/bench/main.cpp:329-332 --
    and the cpu_baseline record of the first `timed` sources)."""
    ref = ref or ReferenceBfs(g.n, g.m, g.flags, g.row_ptr, g.col_idx)
    ref.run(sources[0])  # warm-up
    comp, secs, edges, bad = [], 0.0, 0, None
    for i, s in enumerate(sources):
        d, dt = ref.run(s)
        c = ref.comp_edges(d)
        comp.append(c)
        if i < timed:
            secs += dt
            edges += c
        if i in own:
            same = np.array_equal(own[i], d)
        elif i in hashes:
            same = hashes[i] == depth_hash(d)
        else:
            same = None
        if same is False and bad is None:
            bad = {"source_index": i, "source": int(s)}
    used = min(timed, len(sources))
    cpu = {"value": edges / secs / 1e9, "unit": "GTEPS", "cores": ref.cores, "kind": ref.kind,
           "sample": f"cpu_do alpha=15 beta=18 on all {used} sources of rank 0, {secs:.1f}s"}
    return bad is None, bad, comp, cpu


def max_over_ranks(vals, world):
    """Element-wise maximum of `vals` over all ranks (the slowest rank's times): every
    multi-GPU figure is the whole job's work over the slowest rank's device time.  Works
    with the NCCL process group of a GPU run and with gloo (CPU tests)."""
    vals = [float(v) for v in vals]
    if world <= 1:
        return vals
    import torch
    import torch.distributed as dist
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor(vals, dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return t.tolist()


def measured_traffic(kernel, workload, grid_blocks):
    """DRAM bytes (read + write) per launch of `kernel` on `workload` at a grid of
    `grid_blocks` blocks (None: any; the file lists the option values that give
    the captured grid, 0 being every resident block), as measured by ncu and
    recorded in profiles/roofline_traffic.txt; None when no capture of that
    launch shape is recorded."""
    try:
        with open(os.path.join(ROOT, "profiles", "roofline_traffic.txt")) as f:
            for line in f:
                parts = line.split()
                if line.startswith("#") or len(parts) < 4 or parts[0] != kernel or parts[1] != workload:
                    continue
                if grid_blocks is None or parts[2] == "*" or str(grid_blocks) in parts[2].split(","):
                    return int(parts[3])
    except OSError:
        pass
    return None


def init_dist(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import datetime
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    return world, rank, local


def secondary_workloads(args, local):
    """The other benchmark configurations, measured in the same process after
    the headline (1 GPU): Chung-Lu 20-iteration PageRank and 64-source batch,
    web PageRank to tol 1e-6, road-grid persistent vs plain BFS.  Each is
    checked against the reference's own CPU code; the summary of each line is
    kept (the full lines come from --workload <name>)."""
    import argparse as _a
    import graph_analytics_applesilicon_b200 as G
    sub = _a.Namespace(**vars(args))
    sub.steps, sub.warmup = 5, 3
    out = {}

    def keep(line, keys):
        return {k: line.get(k) for k in keys if k in line}

    common = ("value", "unit", "ms_per_step", "higher_is_better", "config", "e2e", "roofline", "clocks",
              "validated", "validated_sources", "cpu_baseline", "compare")
    t = time.time()
    sub.workload = "road_bfs"
    out["road_bfs"] = keep(bfs_config_workload(sub, 1, 0, local), common)
    sub.workload = "web_pr_tol"
    out["web_pr_tol"] = keep(pagerank_tol_workload(sub, 1, 0, local),
                             ("value", "unit", "config", "e2e", "results", "gs_accuracy_ok", "reference_check",
                              "validated"))
    cl = G.gen.chung_lu(3070000, 2.2, 76.0, 307)
    sub.workload = "chunglu_pr20"
    sub.n = cl.n
    out["chunglu_pr20"] = keep(pagerank_workload(sub, 1, 0, local, g=cl),
                               common + ("accuracy", "reference_check"))
    sub.workload = "chunglu_bfs64"
    out["chunglu_bfs64"] = keep(bfs_config_workload(sub, 1, 0, local, g=cl), common)
    log(f"secondary workloads: {time.time() - t:.1f}s")
    return out


def fixed_options(G, spec, selector):
    """--fixed-opts BLOCK,GRID,HUB: the persistent / batched kernels' launch
    shape and hub cut, given instead of tuned (profiling runs)."""
    block, grid, hub = (int(x) for x in spec.split(","))
    return G.BfsOptions(selector=selector, block=block, grid_blocks=grid, hub_min=hub)


def headline_config(n, m, world, per_rank):
    """The workload description both arms print (identical keys and values)."""
    return {"workload": WORKLOAD, "graph": "rmat scale 22, 8.5*2^22 drawn edges (seed 22), ids permuted (seed 1)",
            "n": n, "m": m, "sources_per_rank": per_rank, "sources_total": per_rank * world,
            "parallelism": f"sources split over {world} GPU(s)" if world > 1 else "1 GPU",
            "l2": "inputs larger than L2 (CSR 293 MB)"}


def reference_arm(args, world, rank):
    """The reference's own CPU BFS (cpu_do, alpha 15 / beta 18, all host
    threads) on the benchmark graph, everything from oracle/_ref: the graph is
    built by the reference's fromEdgeList, reorder "random" and permute from
    the restated quadrant draw, sources by the oracle's pickSources.  This
    library is not imported.  One step = cpu_do over 64 sources (at N > 1 a
    window of 64 of the 64*N sources, rotating per step)."""
    if rank != 0:
        return
    O = _oracle()
    t = time.time()
    if O.ref() is not None:
        rg = O.ref_rmat_graph(SCALE, EDGES_DRAWN, GEN_SEED, PERM_SEED)
        hg = rg.host()
    else:  # the oracle's restatement of the same construction
        rg = None
        hg = O.permute(O.gen("rmat_edges", SCALE, EDGES_DRAWN, 0, GEN_SEED), O.random_perm(1 << SCALE, PERM_SEED))
    srcs_all = O.pick_sources(hg, args.sources * world, 1)
    log(f"reference graph n={hg.n} m={hg.m} built in {time.time() - t:.1f}s")
    ref = ReferenceBfs(hg.n, hg.m, hg.flags, hg.row_ptr, hg.col_idx, ref_graph=rg)
    comp = {}

    def step(i):
        k = len(srcs_all)
        window = [srcs_all[(i * args.sources + j) % k] for j in range(min(args.sources, k))]
        secs, edges = 0.0, 0
        for s in window:
            d, dt = ref.run(s)
            if int(s) not in comp:
                comp[int(s)] = ref.comp_edges(d)
            secs += dt
            edges += comp[int(s)]
        return secs, edges

    for i in range(args.warmup):
        step(i)
    secs = edges = 0
    for i in range(args.steps):
        a, b = step(args.warmup + i)
        secs += a
        edges += b
    v = edges / secs / 1e9
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "GTEPS", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": secs / max(1, args.steps) * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32",
            "data": "synthetic", "config": headline_config(hg.n, hg.m, world, args.sources),
            "cpu_baseline": {"value": v, "unit": "GTEPS", "cores": ref.cores, "kind": ref.kind,
                             "sample": f"cpu_do alpha=15 beta=18, {args.sources} sources per step, "
                                       f"{args.steps} steps, {secs:.1f}s"},
            "e2e": {"value": v, "unit": "GTEPS", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def _timed(fn, reps=1):
    best = float("inf")
    for _ in range(reps):
        t0 = time.perf_counter()
        fn()
        best = min(best, time.perf_counter() - t0)
    return best * 1e3


def bfs_config_workload(args, world, rank, local, g=None):
    """road_bfs: 1400 x 1400 road-shaped grid (4% of edges dropped, 0.5% diagonal
    links, seed 1400; ~1.96M vertices, diameter > 1400 levels); 8 sources,
    single-source persistent BFS vs the per-level plain gpu_do, plus the
    64-source batch in one launch vs 64 plain runs.
    chunglu_bfs64: Chung-Lu graph (3.07M vertices, gamma 2.2, mean degree 76,
    seed 307); one 64-source batch in one launch with the learned batched
    selector and autotuned hub cut / block size, vs 64 plain gpu_do runs.
    Every batch row is checked against the reference's cpu_do, and the TEPS
    denominators come from the reference's depths."""
    import torch
    import graph_analytics_applesilicon_b200 as G
    torch.cuda.set_device(local)
    t = time.time()
    road = args.workload == "road_bfs"
    if g is None:
        g = G.gen.road(1400, 1400, 0.04, 0.005, 1400) if road else G.gen.chung_lu(3070000, 2.2, 76.0, 307)
    log(f"{args.workload}: n={g.n} m={g.m} built in {time.time() - t:.1f}s")
    srcs64 = G.pick_sources_gpu(g, 64, 1)
    bfs = G.GpuBfs(g)
    if args.adjacency == "hub-first":
        bfs.hub_first()  # device layout only: same depths, earlier bottom-up exits
    sel1, sel2 = G.default_selector_params("single"), G.default_selector_params("batch")
    if sel1 is not None:
        bfs.set_selector(sel1, 0)
    if sel2 is not None:
        bfs.set_selector(sel2, 1)
    o1 = G.BfsOptions(selector="learned" if sel1 is not None else "rule")
    o1 = fixed_options(G, args.fixed_opts, o1.selector) if args.fixed_opts else \
        bfs.autotune("gpu_do_persistent", srcs64[:2], o1)
    # the batch runs with whichever selector (learned or the alpha/beta rule)
    # is faster on this graph after tuning block size, hub cut and grid size
    batch_cands = {}
    for sel in (("rule", "learned") if sel2 is not None else ("rule",)):
        if args.fixed_opts:  # profiling runs: the launch shape given, no tuning launches
            if sel == args.selector:
                batch_cands[sel] = (0.0, fixed_options(G, args.fixed_opts, sel))
            continue
        ob_ = bfs.autotune("batch", srcs64, G.BfsOptions(selector=sel))
        bfs.run_batch(srcs64, opts=ob_)
        bfs.run_batch(srcs64, opts=ob_)
        batch_cands[sel] = (bfs.lastGpuMs(), ob_)
    ob = min(batch_cands.values(), key=lambda x: x[0])[1]
    d64 = bfs.run_batch(srcs64, opts=ob)
    batch_levels = bfs.lastLevels()
    for _ in range(args.warmup):
        bfs.run_batch(srcs64, opts=ob)
    with ClockSampler(local) as clocks:
        batch_ms = []
        for _ in range(args.steps):
            bfs.run_batch(srcs64, opts=ob)
            batch_ms.append(bfs.lastGpuMs())
        single = srcs64[:8] if road else srcs64
        single_ms = []
        for s in single:
            bfs.run("gpu_do_persistent", int(s), opts=o1)
            single_ms.append(bfs.lastGpuMs())
        pinned = torch.empty((64, g.n), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
        e2e = _timed(lambda: bfs.run_batch(srcs64, out=pinned, opts=ob), args.steps)
    plain = srcs64[:4] if road else srcs64[:16]
    plain_ms = []
    pb = G.GpuBfs(g) if args.adjacency != "natural" else bfs  # the reference's algorithm, caller's order
    for s in plain:
        pb.run("gpu_do", int(s))
        plain_ms.append(pb.lastGpuMs())
    plain_e2e = [_timed(lambda: pb.run("gpu_do", int(s))) for s in plain[:2]]
    if pb is not bfs:
        pb.close()
    # the single-source forms on a few sources, for the check below
    singles = {i: bfs.run("gpu_do_persistent", int(srcs64[i]), opts=o1) for i in (0, 17, 63)}
    bfs.close()
    batch_t, e2e = max_over_ranks([statistics.median(batch_ms), e2e], world)
    if rank != 0:
        return None
    # every batch row (the e2e call's host output) and the single-source runs
    # against the reference's cpu_do; TEPS denominators from the reference
    valid, bad, comp, cpu = check_against_reference(g, list(srcs64), {i: pinned[i] for i in range(64)}, {})
    valid = valid and all(np.array_equal(d64[i], pinned[i]) and np.array_equal(d, pinned[i])
                          for i, d in singles.items())
    cidx = {int(s): c for s, c in zip(srcs64, comp)}
    e64 = sum(comp)
    single_gteps = sum(cidx[int(s)] for s in single) / (sum(single_ms) * 1e-3) / 1e9
    plain_gteps = sum(cidx[int(s)] for s in plain) / (sum(plain_ms) * 1e-3) / 1e9
    value = world * e64 / (batch_t * 1e-3) / 1e9  # every rank runs its own batch (replicas)
    peak, peak_kind = peaks()
    bytes_per_trav = 4 * (g.n + 1) + 4 * g.m + 4 * g.n
    achieved = 64 * bytes_per_trav / (batch_t * 1e-3) / 1e9
    traffic = measured_traffic("batchBfsKernel", args.workload, ob.grid_blocks)
    dram = traffic / (batch_t * 1e-3) / 1e9 if traffic else None
    line = {"metric": METRIC, "value": value, "unit": "GTEPS", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": batch_t, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "u64 masks / u32 depths", "data": "synthetic",
            "config": {"workload": args.workload, "n": g.n, "m": g.m, "sources": 64, "batch_selector": ob.selector,
                       "adjacency": args.adjacency,
                       "batch_tuning_ms": {k: round(v[0], 3) for k, v in batch_cands.items()},
                       "tuned_block": ob.block, "tuned_hub_min": ob.hub_min, "tuned_grid_blocks": ob.grid_blocks,
                       "single_tuned": {"block": o1.block, "grid_blocks": o1.grid_blocks, "hub_min": o1.hub_min},
                       "parallelism": f"replicas{world}"},
            "e2e": {"value": world * e64 / (e2e * 1e-3) / 1e9, "unit": "GTEPS", "h2d_bytes_per_step": 256,
                    "d2h_bytes_per_step": int(depth_wire_bytes(g.n, batch_levels) * 64 * g.n),
                    "result_bytes_per_step": 4 * 64 * g.n},
            "gpu_launches": args.steps * (1 if road else 2),  # the cluster kernel; the traversal and its rows
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                         "traffic": traffic, "peak_source": peak_kind, "kernel": "batchBfsKernel",
                         "bytes_per_launch": 64 * bytes_per_trav, "mean_launch_ms": batch_t,
                         "note": "graph-pass equivalents: 64 traversals per launch",
                         "dram_achieved": dram, "dram_frac": dram / peak if dram else None},
            "clocks": clocks.summary(), "validated": bool(valid), "validated_sources": 64 if valid else 0,
            "cpu_baseline": cpu,
            "compare": {"batch64_one_launch_gteps": value,
                        "single_source_persistent_gteps": single_gteps,
                        "single_selector": o1.selector,
                        "plain_gpu_do_gteps": plain_gteps,
                        "plain_gpu_do_ms_per_source": statistics.mean(plain_ms),
                        "plain_gpu_do_e2e_ms_per_source": statistics.mean(plain_e2e),
                        "persistent_ms_per_source": statistics.mean(single_ms),
                        "speedup_persistent_vs_plain": statistics.mean(plain_ms) / statistics.mean(single_ms),
                        "speedup_batch_vs_64_plain": 64 * statistics.mean(plain_ms) / batch_t}}
    if bad is not None:
        line["validation_failure"] = bad
    return line


def edge_text(u, v) -> bytes:
    """1-based 'u<TAB>v' lines, formatted with vectorised digit arithmetic."""
    u = np.asarray(u, np.int64) + 1
    v = np.asarray(v, np.int64) + 1
    n, W = u.size, 10
    rows = np.empty((n, 2 * W + 2), np.uint8)
    for col, x in ((0, u), (W + 1, v)):
        d = np.full((n, W), 0xFF, np.uint8)  # 0xFF: no digit (dropped below)
        y = x.copy()
        for k in range(W - 1, -1, -1):
            has = (y > 0) | (k == W - 1)
            d[has, k] = (48 + y[has] % 10).astype(np.uint8)
            y //= 10
        rows[:, col:col + W] = d
    rows[:, W] = 9
    rows[:, 2 * W + 1] = 10
    flat = rows.reshape(-1)
    return flat[flat != 0xFF].tobytes()


def snap_convert_workload(args, world, rank, local):
    """SNAP edge-list text -> CSR (graph::convertSnap, src/graph/snap.cpp:85-149,
    the gconvert path): the undirected edges of the R-MAT scale-22 benchmark
    graph, each written once (u < v) as a 1-based 'u<TAB>v' line (34.6M lines,
    ~0.55 GB of plain text, read from the page cache), converted as undirected
    to a .bin.  value: M edge lines/s of gb_convert_snap_gpu (read, H2D,
    parse, relabel, sort, D2H, .bin write -- so value is also the end-to-end
    number); cpu_baseline: the reference's own convertSnap (oracle/_ref, its
    OpenMP compaction on all host cores) on the same file."""
    import tempfile
    import torch
    import graph_analytics_applesilicon_b200 as G
    torch.cuda.set_device(local)
    g, _ = build_graph(G, nsrc=1)
    rows = np.repeat(np.arange(g.n, dtype=np.int64), np.diff(g.row_ptr.astype(np.int64)))
    keep = rows < g.col_idx
    u, v = rows[keep], g.col_idx[keep].astype(np.int64)
    del rows, keep
    tmp = tempfile.mkdtemp(prefix="snapbench_")
    txt, out = os.path.join(tmp, "rmat22.txt"), os.path.join(tmp, "rmat22.bin")
    t = time.time()
    with open(txt, "wb") as f:
        f.write(b"# R-MAT scale 22 benchmark graph, undirected edges once\n")
        for i in range(0, u.size, 1 << 22):
            f.write(edge_text(u[i:i + (1 << 22)], v[i:i + (1 << 22)]))
    text_bytes, lines = os.path.getsize(txt), int(u.size)
    log(f"snap text: {lines} lines, {text_bytes / 1e9:.2f} GB written in {time.time() - t:.1f}s")
    st = None
    for _ in range(args.warmup):
        st = G.convert_snap_gpu(txt, out, False)
    ts = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        st = G.convert_snap_gpu(txt, out, False)
        ts.append(time.perf_counter() - t0)
    conv = G.load(out)
    # g is symmetric, so the conversion gives back g without its isolated
    # vertices, the rest in the same order (relabelling by increasing raw id)
    deg = np.diff(g.row_ptr.astype(np.int64))
    ok = conv.n == int((deg > 0).sum()) and conv.m == g.m and st["lines"] == lines
    if ok:
        new = np.cumsum(deg > 0) - 1
        ok = (bool(np.array_equal(conv.col_idx, new[g.col_idx].astype(np.uint32)))
              and bool(np.array_equal(np.diff(conv.row_ptr.astype(np.int64)), deg[deg > 0])))
    sec = max_over_ranks([statistics.median(ts)], world)[0]
    value = world * lines / sec / 1e6
    cpu = None
    if rank == 0:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle_py as O
        if O.ref_available():
            t0 = time.perf_counter()
            O.ref_convert_snap(txt, os.path.join(tmp, "ref.bin"), False)
            rs = time.perf_counter() - t0
            cpu = {"value": lines / rs / 1e6, "unit": "M lines/s", "cores": os.cpu_count(), "kind": "reference",
                   "sample": f"graph::convertSnap on the same {text_bytes / 1e9:.2f} GB file, one run, {rs:.1f}s"}
            os.unlink(os.path.join(tmp, "ref.bin"))
    for f in (txt, out):
        os.unlink(f)
    os.rmdir(tmp)
    if rank != 0:
        return None
    line = {"metric": "SNAP text -> CSR .bin conversion (gconvert)", "value": value, "unit": "M lines/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8 text / u32 ids",
            "data": "synthetic", "config": {"workload": "snap_rmat22_text", "lines": lines, "text_bytes": text_bytes,
                                            "n": conv.n, "m": conv.m, "directed": False},
            "e2e": {"value": value, "unit": "M lines/s", "h2d_bytes_per_step": text_bytes,
                    "d2h_bytes_per_step": 4 * (conv.n + 1 + conv.m)},
            "roofline": None, "cpu_baseline": cpu, "validated": ok, "stats": st}
    return line


def pagerank_tol_workload(args, world, rank, local):
    """Web-shaped directed graph (875,000 vertices, geometric out-degree mean
    5.8 -> ~15% dangling, Zipf s=2.1 in-degree, seed 875): PageRank to tol 1e-6,
    Jacobi (degree-adaptive pull) vs in-place Gauss-Seidel (pair deferral K=2),
    FP32 against the FP64 GPU oracle and against the reference's own
    pagerankSerial with checkRanks (Jacobi forms) or gsNoWorseThanJacobi
    (Gauss-Seidel), as gbench --validate does (src/bench/main.cpp:474-495).
    value: ms to tol of the faster method that meets its accuracy rule."""
    import torch
    import graph_analytics_applesilicon_b200 as G
    torch.cuda.set_device(local)
    g = G.gen.web(875000, 5.8, 2.1, 875)
    gin = G.transpose_gpu(g)
    pr = G.GpuPageRank(g.n, g, gin, g.degrees())
    pr.prepareGS(2)
    o = G.PrOptions(tol=1e-6, iters=1000)
    pr.run("gpu_pull_f64", o)
    ref_jac = pr.ranks_f64()
    pr.run("gpu_pull_f64", G.PrOptions(tol=1e-12, iters=2000))
    conv = pr.ranks_f64()
    res, final = {}, {}
    for v in ("gpu_pull_adaptive", "gpu_pull_vector", "gpu_pull_gs"):
        for _ in range(args.warmup):
            pr.run(v, o)
        ts = []
        for _ in range(args.steps):
            r = pr.run(v, o)
            ts.append(r.gpu_ms)
        got = pr.ranks().astype(np.float64)
        final[v] = pr.ranks()
        res[v] = {"ms_to_tol": statistics.median(ts), "iters": r.iters, "last_delta": r.last_delta,
                  "l1_vs_fp64_same_method": float(np.abs(got - ref_jac).sum()),
                  "l1_vs_converged": float(np.abs(got - conv).sum()), "sum": float(got.sum())}
    jac_l1 = float(np.abs(ref_jac - conv).sum())
    gs_ok = res["gpu_pull_gs"]["l1_vs_converged"] <= max(1e-4, jac_l1)
    best = "gpu_pull_gs" if gs_ok and res["gpu_pull_gs"]["ms_to_tol"] < res["gpu_pull_adaptive"]["ms_to_tol"] \
        else "gpu_pull_adaptive"
    res[best]["ms_to_tol"] = max_over_ranks([res[best]["ms_to_tol"]], world)[0]  # the slowest replica
    if rank != 0:
        pr.close()
        return None
    out = torch.empty(g.n, dtype=torch.float32, pin_memory=True).numpy()
    e2e = _timed(lambda: (pr.run(best, o), G.check(G.lib().gb_pr_ranks(pr._h, out))), 3)
    pr.close()
    reference = pagerank_reference_check(gin, g.degrees(), final, 1000, 1e-6)
    valid = reference.get("ok") if reference else None
    line = {"metric": METRIC, "value": res[best]["ms_to_tol"], "unit": "ms to tol 1e-6", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": res[best]["ms_to_tol"],
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f32 (f64 residual)",
            "data": "synthetic", "config": {"workload": "web_pr_tol", "n": g.n, "m": g.m, "method": best},
            "e2e": {"value": e2e, "unit": "ms to tol 1e-6", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 4 * g.n},
            "gpu_launches": None, "results": res, "fp64_jacobi_vs_converged_l1": jac_l1, "gs_accuracy_ok": gs_ok,
            "reference_check": reference, "validated": valid}
    return line


def pagerank_reference_check(gin, outdeg, ranks: dict, iters: int, tol: float, serial=True):
    """The reference's own PageRank (oracle/_ref: pagerankSerial, or
    pagerankOmp with all host threads for the 234M-edge graph -- the same
    per-vertex double sums in parallel) on the full graph, and its checkRanks
    (L1 < 1e-4, top-1000 relative error < 1e-3, |sum - 1| < 1e-4) of every
    FP32 result in `ranks`.  Gauss-Seidel results are held to the reference's
    gsNoWorseThanJacobi against the converged (tol 1e-10) ranks, as gbench
    --validate does.  None when the reference build is absent."""
    O = _oracle()
    if O.ref() is None:
        return None
    rg = O.RefGraph.of(O.HostGraph(gin.n, gin.m, gin.flags, gin.row_ptr, gin.col_idx))
    threads = -1 if serial else 0
    t0 = time.perf_counter()
    ref, it, _ = rg.pagerank(outdeg, iters, tol, threads=threads)
    ref_s = time.perf_counter() - t0
    out = {"reference": ("pagerankSerial" if serial else "pagerankOmp (all threads)") + f", {it} iterations",
           "reference_s": ref_s, "checks": {}}
    ok = True
    conv = jac = None
    for name, r in ranks.items():
        c = O.ref_check_ranks(ref, r)
        rec = {"l1": c.l1, "max_rel_top1000": c.max_rel_top, "sum": c.sum}
        if name == "gpu_pull_gs":
            if conv is None:
                conv, _, _ = rg.pagerank(outdeg, 1000, 1e-10, threads=threads)
                jac = O.check_ranks(conv, ref)  # the Jacobi reference's own distance from convergence
            cg = O.ref_check_ranks(conv, r)
            rec["vs_converged"] = {"l1": cg.l1, "max_rel_top1000": cg.max_rel_top, "sum": cg.sum}
            rec["ok"] = O.gs_no_worse(cg, jac)
        else:
            rec["ok"] = c.ok()
        ok = ok and rec["ok"]
        out["checks"][name] = rec
    out["ok"] = ok
    return out


def pagerank_workload(args, world, rank, local, g=None):
    """Chung-Lu graph (3.07M vertices, gamma 2.2, mean degree 76, seed 307, ids
    permuted): 20 fixed Jacobi iterations in FP32 of the faster of the two
    exact pulls (degree-adaptive, or blocked: contributions staged in shared
    memory), one step = one 20-iteration run (a CUDA-graph replay), ms per
    iteration.
    Checked against the double-precision GPU pull at L1 < 1e-4 and against the
    reference's own pagerankOmp (all host threads, 20 iterations) with its
    checkRanks; that run is also the CPU baseline."""
    import torch
    import graph_analytics_applesilicon_b200 as G
    torch.cuda.set_device(local)
    t = time.time()
    if g is None:
        g = G.gen.chung_lu(args.n, 2.2, 76.0, 307)
    log(f"chung-lu n={g.n} m={g.m} built in {time.time() - t:.1f}s")
    pr = G.GpuPageRank(g.n, g, g, g.degrees())  # undirected: out-CSR = in-CSR
    o = pr.autotune(G.PrOptions(iters=20))  # degree-class cut points and block size
    pr.run("gpu_pull_f64", o)
    ref = pr.ranks_f64()
    # the two exact pulls: degree-adaptive (gathers through L2) and blocked
    # (contributions staged in shared memory); the faster one is the value
    cand, l1s, finals = {}, {}, {}
    for v in ("gpu_pull_adaptive", "gpu_pull_blocked"):
        pr.run(v, o)
        finals[v] = pr.ranks()
        l1s[v] = float(np.abs(finals[v].astype(np.float64) - ref).sum())
        cand[v] = min(pr.run(v, o).gpu_ms for _ in range(3))
    if world > 1:  # every rank runs the same variant
        cand = dict(zip(cand, max_over_ranks(list(cand.values()), world)))
    variant = min(cand, key=cand.get)
    l1 = l1s[variant]
    stream = torch.cuda.ExternalStream(G.lib().gb_pr_stream(pr._h))
    for _ in range(args.warmup):
        pr.run(variant, o)
    barrier = (lambda: (__import__("torch.distributed").distributed.barrier(), torch.cuda.synchronize())) \
        if world > 1 else torch.cuda.synchronize
    barrier()
    with ClockSampler(local) as clocks:
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        gpu = []
        ev0.record(stream)
        for _ in range(args.steps):
            r = pr.run(variant, o)
            gpu.append(r.gpu_ms)
        ev1.record(stream)
        ev1.synchronize()
        total = ev0.elapsed_time(ev1)
        e2e = []
        out = torch.empty(g.n, dtype=torch.float32, pin_memory=True).numpy()
        for _ in range(args.steps):
            t0 = time.perf_counter()
            pr.run(variant, o)
            G.check(G.lib().gb_pr_ranks(pr._h, out))
            e2e.append((time.perf_counter() - t0) * 1e3)
    total, e2e_sum = max_over_ranks([total, sum(e2e)], world)
    compare = {v + "_ms_per_iter": t / 20 for v, t in cand.items()}
    compare.update({v + "_l1_vs_fp64_gpu": x for v, x in l1s.items()})
    for v in ("gpu_pull_vector", "gpu_pull_scalar", "gpu_push"):
        rr = [pr.run(v, o).gpu_ms for _ in range(2)]
        compare[v + "_ms_per_iter"] = min(rr) / 20
    pr.close()
    if rank != 0:
        return None
    ms_iter = total / args.steps / 20
    peak, peak_kind = peaks()
    bytes_sweep = 4 * (g.n + 1) + 8 * g.m + 4 * g.n
    kernel_ms = statistics.mean(gpu) / 20
    achieved = bytes_sweep / (kernel_ms * 1e-3) / 1e9
    cpu, reference = None, None
    if world == 1:
        reference = pagerank_reference_check(g, g.degrees(), finals, 20, 0.0, serial=False)
        if reference is not None and not args.no_cpu_baseline:
            O = _oracle()
            cpu = {"value": reference["reference_s"] * 1e3 / 20, "unit": "ms/iter",
                   "cores": int(O.ref().gref_max_threads()), "kind": "reference",
                   "sample": "cpu_omp (dynamic,256), 20 iterations on the full graph"}
    line = {"metric": METRIC, "value": ms_iter, "unit": "ms/iter", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total / args.steps, "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "chunglu_pr20", "n": g.n, "m": g.m, "variant": variant,
                       "iters": 20, "tuned": {"tg": o.tg, "small_max": o.small_max, "large_min": o.large_min},
                       "parallelism": f"replicas{world}", "l2": "inputs larger than L2 (in-CSR 947 MB)"},
            "e2e": {"value": e2e_sum / args.steps / 20, "unit": "ms/iter", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 4 * g.n},
            "gpu_launches": 21 * args.steps,
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                         "traffic": (measured_traffic("prAdaptiveKernel" if variant == "gpu_pull_adaptive"
                                                      else "prBlockedKernel", "chunglu_pr20", None)
                                     if args.n == 3070000 else None),
                         "peak_source": peak_kind,
                         "kernel": "prAdaptiveKernel" if variant == "gpu_pull_adaptive" else "prBlockedKernel",
                         "bytes_per_launch": bytes_sweep, "mean_launch_ms": kernel_ms},
            "cpu_baseline": cpu, "clocks": clocks.summary(),
            "accuracy": {"l1_vs_fp64_gpu": l1, "ok": l1 < 1e-4}, "reference_check": reference,
            "validated": (l1 < 1e-4) and (reference is None or reference["ok"]), "compare": compare}
    return line


def gather_rows(rows: np.ndarray, world: int) -> list:
    """All ranks' int64 rows (same shape on every rank), in rank order: the
    per-source results of a split batch meet on rank 0 (NCCL on a GPU run,
    gloo in the CPU tests)."""
    if world <= 1:
        return [rows]
    import torch
    import torch.distributed as dist
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.from_numpy(np.ascontiguousarray(rows, np.int64)).to(dev)
    out = [torch.empty_like(t) for _ in range(world)]
    dist.all_gather(out, t)
    return [o.cpu().numpy() for o in out]


def source_rows(depths: np.ndarray, deg: np.ndarray) -> np.ndarray:
    """Per source: (GPU component edges, depth digest as two int64 words)."""
    import concurrent.futures as cf
    with cf.ThreadPoolExecutor(8) as ex:
        digests = list(ex.map(lambda d: depth_hash(d), depths))
    rows = np.zeros((len(depths), 3), np.int64)
    for i, d in enumerate(depths):
        rows[i, 0] = int(deg[d != 0xFFFFFFFF].sum()) // 2
        rows[i, 1:] = np.frombuffer(digests[i], np.int64)
    return rows


def split_sources(srcs_all, world, rank, per_rank):
    """Rank k runs sources [k*per_rank, (k+1)*per_rank) of the 64*N picked
    sources: no source runs twice and rank 0 keeps the single-GPU set."""
    return srcs_all[rank * per_rank:(rank + 1) * per_rank]


def headline_workload(args, world, rank, local):
    import torch
    import graph_analytics_applesilicon_b200 as G
    torch.cuda.set_device(local)
    g, srcs_all = build_graph(G, args.scale, args.sources * world)
    srcs = split_sources(srcs_all, world, rank, args.sources)
    bfs = G.GpuBfs(g)
    if args.adjacency == "hub-first":
        bfs.hub_first()  # device layout only: same depths, earlier bottom-up exits
    sel = G.default_selector_params("single")
    if sel is not None:
        bfs.set_selector(sel, 0)
    # per-graph autotuning of block size, grid size and hub cut for each
    # selector, then the alpha/beta rule judges: the learned selector runs
    # unless the tuned rule is faster on these sources (untimed)
    cands = {}
    for name in (("learned", "rule") if sel is not None else ("rule",)):
        if args.fixed_opts:  # profiling runs: the launch shape given, no tuning launches
            if name != args.selector:
                continue
            o = fixed_options(G, args.fixed_opts, name)
            cands[name] = (0.0, o)
            continue
        o = bfs.autotune("gpu_do_persistent", srcs[:4], G.BfsOptions(selector=name))
        for s_ in srcs[:16]:
            bfs.run("gpu_do_persistent", int(s_), opts=o)
        t_ = 0.0
        for s_ in srcs[:16]:
            bfs.run("gpu_do_persistent", int(s_), opts=o)
            t_ += bfs.lastGpuMs()
        cands[name] = (t_, o)
    if world > 1 and not args.fixed_opts:  # every rank must run the same options
        import torch.distributed as dist
        votes = torch.tensor([cands[k][0] for k in sorted(cands)], dtype=torch.float64, device="cuda")
        dist.all_reduce(votes, op=dist.ReduceOp.SUM)
        selector = sorted(cands)[int(torch.argmin(votes))]
    else:
        selector = min(cands, key=lambda k: cands[k][0])
    opts = cands[selector][1]  # the one-at-a-time judge; the in-flight choice below decides
    stream = torch.cuda.ExternalStream(G.lib().gb_bfs_stream(bfs._h))
    # traversals in flight in one gb_bfs_run_many call (each on 1/K of the
    # resident blocks, its own stream and state): the selector and K of the
    # fastest run_many over this rank's sources, by device time (untimed) --
    # the configuration the timed steps run
    flight_ms = {}
    for name, (_, o_) in cands.items():
        for k in ((args.in_flight,) if args.in_flight else (1, 2, 3, 4, 8, 12, 16)):
            ok = G.BfsOptions(selector=o_.selector, block=o_.block, grid_blocks=0 if k > 1 else o_.grid_blocks,
                              hub_min=o_.hub_min, in_flight=k)
            bfs.run_many("gpu_do_persistent", srcs, opts=ok, device=True)
            t_ = []
            for _ in range(3):
                ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                ev0.record(stream)
                bfs.run_many("gpu_do_persistent", srcs, opts=ok, device=True)
                ev1.record(stream)
                ev1.synchronize()
                t_.append(ev0.elapsed_time(ev1))
            flight_ms[(name, k)] = (min(t_), ok)
    # the batched kernel (64 sources to a launch, per-vertex 64-bit masks) through
    # the same call, tuned per selector on these sources: a candidate like the
    # others, keyed (selector, 0)
    if not args.fixed_opts or args.in_flight == 0:
        sel_b = G.default_selector_params("batch")
        if sel_b is not None:
            bfs.set_selector(sel_b, 1)
        for name in (("learned", "rule") if sel_b is not None else ("rule",)):
            if args.fixed_opts and name != args.selector:
                continue
            ob_ = (fixed_options(G, args.fixed_opts, name) if args.fixed_opts
                   else bfs.autotune("batch", srcs[:64], G.BfsOptions(selector=name)))
            bfs.run_many("batch", srcs, opts=ob_, device=True)
            t_ = []
            for _ in range(3):
                ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                ev0.record(stream)
                bfs.run_many("batch", srcs, opts=ob_, device=True)
                ev1.record(stream)
                ev1.synchronize()
                t_.append(ev0.elapsed_time(ev1))
            flight_ms[(name, 0)] = (min(t_), ob_)
    keys = sorted(flight_ms)
    if world > 1:  # every rank runs the same selector and number in flight
        import torch.distributed as dist
        votes = torch.tensor([flight_ms[k][0] for k in keys], dtype=torch.float64, device="cuda")
        dist.all_reduce(votes, op=dist.ReduceOp.SUM)
        best = keys[int(torch.argmin(votes))]
    else:
        best = min(keys, key=lambda k: flight_ms[k][0])
    selector, in_flight = best
    opts = flight_ms[best][1]
    head_variant = "batch" if in_flight == 0 else "gpu_do_persistent"

    max_levels = 0  # sets the packed depth width on the PCIe wire
    for s in srcs:
        bfs.run("gpu_do_persistent", int(s), opts=opts)
        max_levels = max(max_levels, bfs.lastLevels())

    def device_step(variant=head_variant, o=opts, h=bfs):
        # one gb_bfs_run_many call: the persistent traversals follow one
        # another on the stream; gpu_do keeps its per-source host loop
        st = stream if h is bfs else torch.cuda.ExternalStream(G.lib().gb_bfs_stream(h._h))
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record(st)
        _, ms, _ = h.run_many(variant, srcs, opts=o, device=True)
        ev1.record(st)
        ev1.synchronize()
        return ev0.elapsed_time(ev1), [float(x) for x in ms]

    pinned = torch.empty(g.n, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    distinct = np.zeros((len(srcs), g.n), np.uint32)  # 1 GB: every source's depths kept

    def e2e_step(out=pinned, stride=0):
        # every source's depths reach host memory (uint32, packed on the wire);
        # stride 0: one buffer reused by every source, as the reference's loop
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        bfs.run_many(head_variant, srcs, out=out, stride=stride, opts=opts)
        return (time.perf_counter() - t0) * 1e3

    def barrier():
        if world > 1:
            import torch.distributed as dist
            dist.barrier()
        torch.cuda.synchronize()

    for _ in range(args.warmup):
        device_step()
        e2e_step()
        e2e_step(distinct, g.n)
    barrier()
    with ClockSampler(local) as clocks:
        step_ms, launch_ms = [], []
        for _ in range(args.steps):
            t, ms = device_step()
            step_ms.append(t)
            launch_ms += ms
        barrier()
        e2e_ms = [e2e_step() for _ in range(args.steps)]
        barrier()
        e2e_distinct_ms = [e2e_step(distinct, g.n) for _ in range(args.steps)]
        barrier()
    total_ms, e2e_total, e2e_distinct_total = max_over_ranks([sum(step_ms), sum(e2e_ms), sum(e2e_distinct_ms)],
                                                             world)
    # the last timed step left every source's depths in `distinct` (the output
    # of the public call): their digests meet on rank 0 for the reference check
    deg = np.diff(g.row_ptr.astype(np.int64))
    rows = gather_rows(source_rows(distinct, deg), world)

    # comparison forms on the same sources (not part of the timed region)
    plain_ms = rule_ms = learned_ms = float("nan")
    rule_opts = None
    if not args.no_compare:
        # the reference's algorithm (plain gpu_do) on the caller's adjacency order
        plain = G.GpuBfs(g) if args.adjacency != "natural" else bfs
        device_step("gpu_do", G.BfsOptions(), plain)
        plain_ms = device_step("gpu_do", G.BfsOptions(), plain)[0]
        if plain is not bfs:
            plain.close()
        # each selector in the same kernel, tuned the same way
        rule_opts = cands["rule"][1] if "rule" in cands else opts
        device_step("gpu_do_persistent", rule_opts)
        rule_ms = device_step("gpu_do_persistent", rule_opts)[0]
        if "learned" in cands:
            device_step("gpu_do_persistent", cands["learned"][1])
            learned_ms = device_step("gpu_do_persistent", cands["learned"][1])[0]
    if rank != 0:
        return None

    # every depth array of every rank against the reference's cpu_do, bit for
    # bit; the TEPS denominators come from the reference's depths
    own = {i: distinct[i] for i in range(len(srcs))}
    hashes = {r * len(srcs) + i: rows[r][i, 1:].tobytes() for r in range(world) for i in range(len(srcs))}
    gpu_comp = [int(x) for r in range(world) for x in rows[r][:, 0]]
    if args.no_validate:
        valid, bad, comp, cpu = None, None, gpu_comp, None
    else:
        valid, bad, comp, cpu = check_against_reference(g, srcs_all, own, hashes, timed=len(srcs))
        valid = valid and comp == gpu_comp
    edges_per_rank_step = sum(comp[:len(srcs)])
    edges_all = sum(comp)
    # reference summary: harmonic mean over sources of per-source GTEPS (src/bench/main.cpp:366-370)
    hmean = len(srcs) / sum((lm * 1e-3) / (c / 1e9) for lm, c in zip(launch_ms[: len(srcs)], comp) if c)

    peak, peak_kind = peaks()
    bytes_per_trav = 4 * (g.n + 1) + 4 * g.m + 4 * g.n
    step_s = statistics.mean(step_ms) * 1e-3
    batched = head_variant == "batch"
    launches_per_step = (len(srcs) + 63) // 64 if batched else len(srcs)
    # a batched launch's time is shared evenly over its sources in launch_ms
    mean_launch = statistics.mean(launch_ms) * (len(srcs) / launches_per_step if batched else 1)
    # graph-pass equivalents: every traversal's algorithmic bytes over the
    # step's device time (launches overlap when in_flight > 1; memsets and gaps
    # between launches count against it)
    pass_rate = bytes_per_trav * len(srcs) / step_s / 1e9
    if batched:
        kernel = f"batchBfsKernel<{opts.block or 512}>"
        traffic = measured_traffic(kernel, WORKLOAD, opts.grid_blocks) if args.scale == SCALE else None
    else:
        kernel = f"persistentBfsKernel<{opts.block or 512}>"
        traffic = (measured_traffic(kernel, WORKLOAD, opts.grid_blocks if opts.in_flight <= 1 else f"x{opts.in_flight}")
                   if args.scale == SCALE else None)
    dram_rate = traffic * launches_per_step / step_s / 1e9 if traffic else None
    # achieved: graph-pass equivalents per second, the algorithmic figure (for
    # the batched kernel, which reads each edge once per level for all 64
    # sources, it can pass the peak); dram_achieved: what ncu measured per launch
    achieved = pass_rate

    value = edges_all * args.steps / (total_ms * 1e-3) / 1e9
    e2e_value = edges_all * args.steps / (e2e_total * 1e-3) / 1e9
    e2e_distinct = edges_all * args.steps / (e2e_distinct_total * 1e-3) / 1e9
    wire = int(depth_wire_bytes(g.n, max_levels) * g.n * len(srcs))
    config = headline_config(g.n, g.m, world, len(srcs))
    if args.scale != SCALE:
        config["workload"] = f"rmat{args.scale}_bfs{len(srcs)}"
    line = {
        "metric": METRIC, "value": value, "unit": "GTEPS", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
        "config": config,
        "method": {"selector": selector, "adjacency": args.adjacency,
                   "tuned": {"block": opts.block, "grid_blocks": opts.grid_blocks, "hub_min": opts.hub_min,
                             "in_flight": opts.in_flight},
                   "variant": head_variant,
                   "step_ms_by_selector_in_flight": {f"{k[0]}/{k[1]}": round(v[0], 3) for k, v in flight_ms.items()},
                   "in_flight_0": "the batched kernel (64 sources to a launch, per-vertex 64-bit masks)",
                   "call": ("gb_bfs_run_many with the batched kernel: one launch per 64 sources, then each "
                            "source's row packed, copied and widened" if batched else
                            "gb_bfs_run_many, one persistent launch per source; in_flight of them at once, "
                            "each on 1/in_flight of the resident blocks")},
        "work": {"edges_per_step": edges_all, "edges_per_step_rank0": edges_per_rank_step,
                 "teps_denominators": "component edges of the reference's cpu_do depths"},
        "e2e": {"value": e2e_value, "unit": "GTEPS", "h2d_bytes_per_step": 4 * len(srcs),
                "d2h_bytes_per_step": wire, "result_bytes_per_step": 4 * g.n * len(srcs),
                "host_output": "one pinned uint32[n] array reused by every source (as the reference's loop)"},
        "e2e_distinct_buffers": {"value": e2e_distinct, "unit": "GTEPS", "h2d_bytes_per_step": 4 * len(srcs),
                                 "d2h_bytes_per_step": wire, "result_bytes_per_step": 4 * g.n * len(srcs),
                                 "host_output": "a separate uint32[n] array per source (1 GB per step)"},
        # a batch: the traversal, its rows and, end to end, a pack for each row (1 MB or more)
        "gpu_launches": launches_per_step * (2 if batched else 1) * args.steps,
        "gpu_launches_e2e": (launches_per_step * (2 if batched else 1) + len(srcs)) * args.steps,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak if achieved else None, "traffic": traffic, "peak_source": peak_kind,
                     "kernel": kernel, "bytes_per_launch": bytes_per_trav,
                     "mean_launch_ms": mean_launch, "launches_at_once": 1 if batched else opts.in_flight,
                     "achieved_basis": "B_bfs = 4(n+1)+4m+4n per traversal x traversals of the step / device "
                                       "step time (graph-pass equivalents; a batched launch reads each edge once "
                                       "per level for all its sources, so this can pass the peak)",
                     "dram_achieved": dram_rate,
                     "dram_frac": dram_rate / peak if dram_rate else None},
        "cpu_baseline": cpu if world == 1 else None,
        "clocks": clocks.summary(),
        "validated": valid,
        "validated_sources": (len(srcs_all) if valid else 0) if valid is not None else None,
        "validation": ("every source's depths (from the timed e2e call) equal "
                       + ("the reference's cpu_do (oracle/_ref)" if cpu and cpu["kind"] == "reference"
                          else "the oracle's cpu_do (oracle/oracle.c)")
                       + " bit for bit" + ("; other ranks' by 128-bit digest" if world > 1 else "")),
        "compare": {"plain_gpu_do_gteps": edges_per_rank_step / (plain_ms * 1e-3) / 1e9,
                    "persistent_rule_gteps": edges_per_rank_step / (rule_ms * 1e-3) / 1e9,
                    "persistent_rule_tuned": ({"block": rule_opts.block, "grid_blocks": rule_opts.grid_blocks,
                                               "hub_min": rule_opts.hub_min} if rule_opts is not None else None),
                    "persistent_learned_gteps": edges_per_rank_step / (learned_ms * 1e-3) / 1e9,
                    "speedup_learned_vs_rule": rule_ms / learned_ms,
                    "speedup_learned_vs_rule_at_in_flight": (
                        flight_ms[("rule", in_flight)][0] / flight_ms[("learned", in_flight)][0]
                        if ("rule", in_flight) in flight_ms and ("learned", in_flight) in flight_ms else None),
                    "judge_ms_16_sources": {k: round(v[0], 4) for k, v in cands.items()},
                    "speedup_vs_plain_gpu_do": plain_ms / (total_ms / args.steps),
                    "hmean_gteps_per_source_launch": hmean,
                    "hmean_note": "harmonic mean of per-source GTEPS from each launch's device time (a batched launch's time shared over its sources) "
                                  "(src/bench/main.cpp:366-370); launches overlap when in_flight > 1"},
    }
    if bad is not None:
        line["validation_failure"] = bad
    return line


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-compare", action="store_true", help="skip the plain/rule comparison runs")
    ap.add_argument("--no-secondary", action="store_true",
                    help="skip the other benchmark configurations (road, Chung-Lu, web) after the headline")
    ap.add_argument("--no-validate", action="store_true",
                    help="skip the reference check of every depth array (profiling runs only; "
                         "the line then says validated: null)")
    ap.add_argument("--fixed-opts", default="",
                    help="BLOCK,GRID,HUB: run the persistent / batched kernels with this launch shape and hub cut "
                         "instead of autotuning (profiling runs)")
    ap.add_argument("--in-flight", type=int, default=0, choices=range(17),
                    help="traversals at once in gb_bfs_run_many (0: measure 1, 2, 3, 4, 8, 12, 16 and keep the "
                         "fastest)")
    ap.add_argument("--selector", default="rule", choices=["rule", "learned"],
                    help="with --fixed-opts: the per-level selector")
    ap.add_argument("--scale", type=int, default=SCALE, help="R-MAT scale (smaller: profiling cases)")
    ap.add_argument("--sources", type=int, default=NSRC, help="sources per GPU")
    ap.add_argument("--workload", default=WORKLOAD,
                    choices=[WORKLOAD, "chunglu_pr20", "road_bfs", "chunglu_bfs64", "web_pr_tol", "snap_convert"],
                    help="rmat22_bfs64 (default, the headline); chunglu_pr20, road_bfs, chunglu_bfs64, web_pr_tol, "
                         "snap_convert")
    ap.add_argument("--n", type=int, default=3070000, help="chunglu_pr20: vertices")
    ap.add_argument("--adjacency", default="hub-first", choices=["hub-first", "natural"],
                    help="BFS device adjacency layout (hub-first: lists by descending neighbour degree; same depths)")
    args = ap.parse_args()
    world, rank, local = init_dist(args)
    if args.impl == "reference":
        reference_arm(args, world, rank)
        return
    args.warmup = max(3, args.warmup)
    workloads = {"chunglu_pr20": pagerank_workload, "road_bfs": bfs_config_workload,
                 "chunglu_bfs64": bfs_config_workload, "web_pr_tol": pagerank_tol_workload,
                 "snap_convert": snap_convert_workload, WORKLOAD: headline_workload}
    line = workloads[args.workload](args, world, rank, local)
    if line is None:
        return
    ok = line.get("validated") is not False
    if args.workload == WORKLOAD and world == 1 and not args.no_secondary:
        line["secondary"] = secondary_workloads(args, local)
        ok = ok and all(v.get("validated") is not False for v in line["secondary"].values())
    print(json.dumps(line), flush=True)
    if not ok:
        log("VALIDATION FAILED: " + json.dumps(line.get("validation_failure")))
        sys.exit(1)


if __name__ == "__main__":
    main()
