"""Benchmark: sequential Gaussian simulation throughput (nodes x realizations / s).

One step = one complete simulation of the workload on the GPU: neighbour
search (kernel a), dependency levels, kriging build + solve (kernel b) and
the level-scheduled sweep over all realizations (kernel c), from the
problem already resident in HBM.  Default workload: 3D 200x200x100 grid
(4M nodes), 5,000 data, exponential variogram with ranges 50/25/5 and a
30 degree rotation, nugget 0.05, search ellipsoid = the variogram's,
maxneighbors 48, 256 realizations, RandomPath seed 4, seeded on-device
standard normals.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Under torchrun each rank simulates its own 256 realizations on its own GPU
(replicas: weak scaling, no collective on the data path).
`--impl reference` times the FP64 CPU restatement of the reference's SEQSIM
(oracle/, all host threads) on a bounded sample of the same workload.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "geostatsprocesses.jl_gb300"))

METRIC = "SGS nodes×reals/s on 1 GB300: learned+FP32 vs plain FP64 path at ≤1e-6 rel err"
UNIT = "nodes*reals/s"


PEAKS_SRC = os.path.join(ROOT, "bench_peaks.cu")
PEAKS_PATH = os.path.join(ROOT, "_build", "libgeosgs_peaks.so")


def build_peaks(force: bool = False) -> str:
    """Compile the throughput probes (bench_peaks.cu) into their own library
    with the product's nvcc flags; measurement infrastructure, outside the
    product's C ABI."""
    sys.path.insert(0, os.path.join(ROOT, "geostatsprocesses.jl_gb300"))
    from geosgs import _build

    if not force and os.path.exists(PEAKS_PATH) and os.path.getmtime(PEAKS_SRC) <= os.path.getmtime(PEAKS_PATH):
        return PEAKS_PATH
    os.makedirs(os.path.dirname(PEAKS_PATH), exist_ok=True)
    tmp = PEAKS_PATH + ".tmp"
    cmd = [_build._nvcc(), *_build.NVCC_FLAGS, "-shared", "-o", tmp, PEAKS_SRC]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {PEAKS_SRC}:\n{r.stderr}")
    os.replace(tmp, PEAKS_PATH)
    return PEAKS_PATH


def measure_peaks() -> dict:
    """FP32 FFMA and FP64 DFMA rates, the Gauss-Jordan pattern rate and the
    device-to-page-locked-host write rate, from the probe library; empty
    where it cannot be built or loaded."""
    out = {}
    try:
        lib = ctypes.CDLL(build_peaks())
    except (OSError, RuntimeError):
        return out
    for name in ("geosgs_peak_fp32", "geosgs_peak_fp64", "geosgs_peak_gj_pattern"):
        getattr(lib, name).argtypes = [ctypes.POINTER(ctypes.c_double)]
    lib.geosgs_peak_host_write.argtypes = [ctypes.c_int64, ctypes.POINTER(ctypes.c_double)]
    lib.geosgs_peak_d2h_copy.argtypes = [ctypes.c_int64, ctypes.POINTER(ctypes.c_double)]
    v = ctypes.c_double(0.0)
    if lib.geosgs_peak_fp32(ctypes.byref(v)) == 0:
        out["fp32_tflops"] = v.value
    if lib.geosgs_peak_fp64(ctypes.byref(v)) == 0:
        out["fp64_tflops"] = v.value
    if lib.geosgs_peak_gj_pattern(ctypes.byref(v)) == 0:
        out["gj_pattern_tflops"] = v.value
    if lib.geosgs_peak_host_write(ctypes.c_int64(1 << 30), ctypes.byref(v)) == 0:
        out["host_write_gbs"] = v.value
    if lib.geosgs_peak_d2h_copy(ctypes.c_int64(1 << 30), ctypes.byref(v)) == 0:
        out["d2h_copy_gbs"] = v.value
    return out


def solve_flops(sizes, refine_steps: int) -> float:
    """Algorithmic FLOPs of the kriging systems, counted for a Cholesky-based
    solve whatever algorithm runs, per system of n neighbours: n(n+1)/2 covariance evaluations, n^3/3 for the
    Cholesky factorization, 2 n^2 for the two triangular solves, per
    refinement step 2 n^2 (residual) + 2 n^2 (correction), 2 n for the
    variance; sizes[n] = number of systems with n neighbours."""
    nn = np.arange(len(sizes), dtype=np.float64)
    per = nn * (nn + 1) / 2 + nn ** 3 / 3 + 2 * nn ** 2 + refine_steps * 4 * nn ** 2 + 2 * nn
    return float(np.sum(np.asarray(sizes, dtype=np.float64) * per))


def config_of(wl, ws: int) -> dict:
    """The workload's configuration, identical for every arm (GPU and
    reference): what is simulated, not how."""
    N, R = wl.domain.nelements(), wl.nreals
    return {"workload": wl.name, "grid": list(wl.domain.dims), "nodes": N,
            "ndata": 0 if wl.data is None else wl.data.nrow(), "maxneighbors": wl.method.maxneighbors,
            "nreals": R, "parallelism": f"replicas x{ws}",
            "l2": "inputs larger than L2 (value array >= %.1f GB)" % (N * R * 4 / 1e9)}


def batch_config_of(bw, ws: int) -> dict:
    N = bw.nodes()
    return {"workload": bw.name, "ndomains": len(bw.items), "nodes": N, "nreals": bw.nreals,
            "ndata": int(sum(0 if w.data is None else w.data.nrow() for w in bw.items)),
            "parallelism": f"replicas x{ws}",
            "l2": "inputs larger than L2 (value array >= %.1f GB)" % (N * bw.nreals * 4 / 1e9)}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="c3", choices=["c1", "c2", "c3", "c4", "c5"])
    ap.add_argument("--ndomains", type=int, default=1000, help="c5: domains in the batch")
    ap.add_argument("--nreals", type=int, default=None)
    ap.add_argument("--no-fp64", action="store_true", help="skip the plain FP64 path measurement")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--cpu-nodes", type=int, default=60000, help="oracle sample size (nodes)")
    ap.add_argument("--no-learned", action="store_true", help="skip training and timing the learned warm start")
    ap.add_argument("--learned-systems", type=int, default=None,
                    help="training systems for the warm start (default 600,000; 10,000,000 for c4)")
    ap.add_argument("--learned-epochs", type=int, default=8)
    ap.add_argument("--sweep-config", default=None,
                    help='JSON sweep configuration (sgs_sweep_config fields) instead of the autotuner, e.g. '
                         '\'{"mode": 0, "lanes_w": 32, "tight": 1}\' (profiling one form)')
    ap.add_argument("--grid", default=None, help="override the 3D grid, e.g. 200,200,50 (profiling a smaller case)")
    ap.add_argument("--ndata", type=int, default=None, help="override the number of data (with --grid)")
    return ap.parse_args()


def workload(name, precision, nreals, grid=None, ndata=None):
    from geosgs import workloads

    if name == "c1":
        wl = workloads.c1(precision)
    elif name == "c2":
        wl = workloads.c2(precision)
    elif name == "c4":
        wl = workloads.c4(precision, dims=tuple(int(x) for x in grid.split(",")) if grid else (256, 256, 256))
    elif grid:
        dims = tuple(int(x) for x in grid.split(","))
        wl = workloads.c3(precision, dims=dims, ndata=ndata if ndata is not None else 5000)
    else:
        wl = workloads.c3(precision)
    if nreals:
        wl.nreals = nreals
    return wl


# ----------------------------------------------------------------- clocks
class ClockSampler:
    """nvidia-smi samples of SM clock and throttle reasons during the timed region."""

    FIELDS = ("uuid,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, uuid: str | None):
        self.uuid = uuid
        self.rows = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
            return self
        self.t = threading.Thread(target=self._read, daemon=True)
        self.t.start()
        return self

    def _read(self):
        for line in self.proc.stdout:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) == 9 and (self.uuid is None or self.uuid in parts[0]):
                self.rows.append(parts)

    def stop(self):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self.rows for i in range(4) if r[5 + i] == "Active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


# ------------------------------------------------------------- distributed
def dist_setup(args):
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import torch.distributed as dist

        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group("gloo")
    return ws, rank, local


def replica_seed(seed: int) -> int:
    """Seed of this rank's realizations: replicas draw disjoint Philox
    streams, so N ranks produce N x R distinct realizations."""
    return seed + int(os.environ.get("RANK", "0")) * 1_000_003


def barrier(ws):
    if ws > 1:
        import torch.distributed as dist

        dist.barrier()


def max_over_ranks(ws, x):
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist

    t = torch.tensor([x], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ---------------------------------------------------------------- CPU leg
def cpu_sample(wl, nodes: int, nthreads: int = 0):
    """FP64 oracle on a bounded sample of the workload: search + solve of
    `nodes` path ranks spread over the whole path, and the draw loop of the
    first `nodes` path ranks for all realizations.  Returns nodes*reals/s."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import geosgs
    import oracle

    oracle.build()
    p, keep = geosgs.build_problem(wl.process, wl.domain, wl.data, wl.method)
    O = oracle.OraclePlan(p, keep)
    N, R = O.N, wl.nreals
    stride = max(1, N // nodes)
    t0 = time.perf_counter()
    O.search(oracle.TEMPLATE, stride=stride, nthreads=nthreads)
    O.solve(stride=stride, nthreads=nthreads)
    t_ss = time.perf_counter() - t0
    n_ss = (N + stride - 1) // stride
    M = min(N, nodes)
    O.search(oracle.TEMPLATE, t1=M, nthreads=nthreads)
    O.solve(t1=M, nthreads=nthreads)
    t0 = time.perf_counter()
    O.simulate(R, None, seed=1, t_end=M, nthreads=nthreads)
    t_sw = time.perf_counter() - t0
    per_node = t_ss / n_ss + t_sw / M  # seconds per node for all R realizations
    cores = nthreads or os.cpu_count()
    sample = (f"oracle FP64 on {wl.name}: search+solve of {n_ss} path ranks (every {stride}th) "
              f"+ draw loop of the first {M} ranks x {R} realizations; {cores} threads")
    return R / per_node, cores, sample, t_ss + t_sw


def run_reference(args):
    """The reference arm: the FP64 CPU restatement of SEQSIM on the host
    cores, each step a bounded sample of the workload (the Julia reference
    has no toolchain on the box).  `value` is the throughput measured on the
    sample; `ms_per_step` is the sample's own wall time; the line says that the
    value is extrapolated from a sample and how large the sample was."""
    ws, rank, _ = dist_setup(args)
    if rank != 0:
        return
    note = ("Julia reference not runnable on this box (no Julia toolchain); timed the FP64 C++ "
            "restatement of SEQSIM (oracle/) instead")
    if args.workload == "c5":
        from geosgs import workloads

        bw = workloads.c5("fp64", nreals=args.nreals or 8, ndomains=args.ndomains)
        vals, secs = [], []
        for i in range(args.warmup + args.steps):
            v, cores, sample, t = cpu_sample_batch(bw, args.cpu_nodes * 4)
            if i >= args.warmup:
                vals.append(v)
                secs.append(t)
        value = statistics.median(vals)
        config = batch_config_of(bw, args.gpus)
        full_ms = 1e3 * bw.nodes() * bw.nreals / value
    else:
        wl = workload(args.workload, "fp64", args.nreals, args.grid, args.ndata)
        vals, secs = [], []
        for i in range(args.warmup + args.steps):
            v, cores, sample, t = cpu_sample(wl, args.cpu_nodes)
            if i >= args.warmup:
                vals.append(v)
                secs.append(t)
        value = statistics.median(vals)
        config = config_of(wl, args.gpus)
        full_ms = 1e3 * wl.domain.nelements() * wl.nreals / value
    out = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * statistics.median(secs),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded PCG64 grid data, path and Philox normals)",
        "config": config,
        "extrapolated": True,
        "sample": sample,
        "sample_wall_ms_per_step": 1e3 * statistics.median(secs),
        "full_workload_ms_estimate": full_ms,
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "note": note,
    }
    print(json.dumps(out))


# --------------------------------------------------------------- GPU legs
def time_device(wl, args, torch, ws, network=None):
    """Device-resident steps: prepare (search, levels, solve) + sweep."""
    import geosgs

    p, keep = geosgs.build_problem(wl.process, wl.domain, wl.data, wl.method)
    plan = geosgs.Plan(p, keep)
    if network is not None:
        plan.set_network(network)
    R = wl.nreals
    Rp = (R + 3) // 4 * 4
    stream = torch.cuda.current_stream().cuda_stream
    # sweep autotuner: once per plan, outside the timed region
    plan.prepare()
    dt = torch.float64 if plan.values_fp64() else torch.float32
    V = torch.empty(plan.N * Rp, dtype=dt, device="cuda")

    def step(i):
        plan.prepare()
        plan.simulate_device(R, None, replica_seed(1000 + i), V, stream)

    if args.sweep_config:
        plan.set_sweep(**json.loads(args.sweep_config))
        sweep_cfg, sweep_tried = dict(plan.sweep_config()), []
    else:
        sweep_cfg, sweep_tried = plan.tune_sweep(R)
    for i in range(args.warmup):
        step(i)
    torch.cuda.synchronize()
    launches0 = plan.info().launches
    sweeps, solves, searches, levels = [], [], [], []
    barrier(ws)
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for i in range(args.steps):
        step(args.warmup + i)
        inf = plan.info()  # waits for this step's sweep to time it
        sweeps.append(inf.ms_sweep)
        solves.append(inf.ms_solve)
        searches.append(inf.ms_search)
        levels.append(inf.ms_levels)
    e1.record()
    torch.cuda.synchronize()
    barrier(ws)
    ms = e0.elapsed_time(e1) / args.steps
    inf = plan.info()
    # kriging-system sizes (grid + data neighbours of every node that solved
    # a system), after the timed region: the solve's algorithmic FLOPs
    cnt = np.empty(plan.N, dtype=np.int32)
    st = np.empty(plan.N, dtype=np.int32)
    plan._check(plan.lib.sgs_plan_neighbors(plan.h, None, cnt.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))))
    plan._check(plan.lib.sgs_plan_weights(plan.h, None, None, st.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))))
    sizes = np.bincount(cnt[st == 0], minlength=plan.k + 1)
    res = dict(ms=max_over_ranks(ws, ms), launches=(inf.launches - launches0), info=inf,
               sweep_config=sweep_cfg, sweep_tried=sweep_tried,
               ms_sweep=statistics.mean(sweeps), ms_solve=statistics.mean(solves),
               ms_search=statistics.mean(searches), ms_levels=statistics.mean(levels),
               system_sizes=sizes)
    plan.close()
    del V
    return res


def time_e2e(wl, args, torch, ws, steps, sweep=None, network=None):
    """Through the public C ABI with host buffers: create (host -> device
    copies of the problem), prepare, simulate with the FP64 result copied to
    pinned host memory, destroy."""
    import geosgs

    N, R = wl.domain.nelements(), wl.nreals
    out = torch.empty((R, N), dtype=torch.float64, pin_memory=True).numpy()
    p, keep = geosgs.build_problem(wl.process, wl.domain, wl.data, wl.method)

    split = {"create": 0.0, "prepare": 0.0, "simulate": 0.0, "destroy": 0.0}

    def step(i):
        t = time.perf_counter()
        plan = geosgs.Plan(p, keep)
        if network is not None:
            plan.set_network(network)
        if sweep:
            plan.set_sweep(**sweep)
        t1 = time.perf_counter()
        plan.prepare()
        t2 = time.perf_counter()
        plan._check(plan.lib.sgs_plan_simulate(plan.h, R, None, replica_seed(77 + i),
                                               out.ctypes.data_as(__import__("ctypes").POINTER(__import__("ctypes").c_double))))
        t3 = time.perf_counter()
        inf = plan.info()
        plan.close()
        t4 = time.perf_counter()
        if i > 0:
            for k_, v_ in zip(split, (t1 - t, t2 - t1, t3 - t2, t4 - t3)):
                split[k_] += v_
        return inf

    step(0)
    barrier(ws)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    infs = [step(1 + i) for i in range(steps)]
    torch.cuda.synchronize()
    dt = max_over_ranks(ws, (time.perf_counter() - t0) / steps)
    time_e2e.split_ms = {k_: round(1e3 * v_ / steps, 2) for k_, v_ in split.items()}
    return dt, infs[-1], float(out[0, :8].sum())


# ------------------------------------------------------- batch of domains
def time_batch(bw, args, torch, ws, precision):
    """Device-resident steps of a batch: prepare (graph: search, levels,
    order, bins, solves) + seeded sweep (graph) into a device array."""
    import geosgs

    probs = []
    for w in bw.items:
        w.method.precision = precision
        probs.append(geosgs.build_problem(w.process, w.domain, w.data, w.method))
    t0 = time.perf_counter()
    B = geosgs.Batch(probs)
    t_create = time.perf_counter() - t0
    R = bw.nreals
    Rp = (R + 3) // 4 * 4
    B.prepare()
    dt = torch.float64 if B.values_fp64() else torch.float32
    V = torch.empty(B.nnodes * Rp, dtype=dt, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    if args.sweep_config:
        B.set_sweep(**json.loads(args.sweep_config))
        cfg, tried = json.loads(args.sweep_config), []
    else:
        cfg, tried = B.tune_sweep(R)

    def step(i):
        B.prepare()
        B.simulate_device(R, replica_seed(1000 + i), V, stream)

    for i in range(args.warmup):
        step(i)
    torch.cuda.synchronize()
    launches0, graphs0 = B.info().launches, B.info().graph_launches
    ph = {"search": [], "levels": [], "solve": [], "sweep": []}
    barrier(ws)
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for i in range(args.steps):
        step(args.warmup + i)
        inf = B.info()
        ph["search"].append(inf.ms_search)
        ph["levels"].append(inf.ms_levels)
        ph["solve"].append(inf.ms_solve)
        ph["sweep"].append(inf.ms_sweep)
    e1.record()
    torch.cuda.synchronize()
    barrier(ws)
    ms = e0.elapsed_time(e1) / args.steps
    inf = B.info()
    # nodes of the domains that keep FP64 values (the sweep's value rows are
    # 8 bytes per realization there, 4 elsewhere)
    n_fp64 = int(sum(int(B.sizes[d]) for d in range(len(B.sizes)) if B.domain_values_fp64(d)))
    res = dict(ms=max_over_ranks(ws, ms), launches=inf.launches - launches0, graphs=inf.graph_launches - graphs0,
               info=inf, sweep_config=cfg, sweep_tried=tried, s_create=t_create, nodes_fp64=n_fp64,
               phases={k: statistics.mean(v) for k, v in ph.items()})
    B.close()
    del V
    torch.cuda.empty_cache()
    return res, probs


def cpu_sample_batch(bw, budget_nodes: int):
    """FP64 oracle on the first domains of the batch (whole domains, up to
    about budget_nodes nodes): nodes*reals/s over the sample."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import geosgs
    import oracle

    oracle.build()
    nodes, secs, used = 0, 0.0, 0
    for w in bw.items:
        n = w.domain.nelements()
        if used and nodes + n > budget_nodes:
            continue
        w.method.precision = "fp64"
        p, keep = geosgs.build_problem(w.process, w.domain, w.data, w.method)
        O = oracle.OraclePlan(p, keep)
        t0 = time.perf_counter()
        O.prepare()
        O.simulate(bw.nreals, None, seed=1)
        secs += time.perf_counter() - t0
        nodes += n
        used += 1
        if nodes >= budget_nodes:
            break
    cores = os.cpu_count()
    sample = (f"oracle FP64 on {used} whole domains of {bw.name} ({nodes} nodes x {bw.nreals} realizations: "
              f"search, solve and draw loop); {cores} threads")
    return nodes * bw.nreals / secs, cores, sample, secs


def main_batch(args, torch, ws, rank, uuid):
    from geosgs import workloads

    bw = workloads.c5("fp32", nreals=args.nreals or 8, ndomains=args.ndomains)
    N, R = bw.nodes(), bw.nreals
    clocks = ClockSampler(uuid).start()
    fast, probs = time_batch(bw, args, torch, ws, "fp32")
    clk = clocks.stop()
    fp64 = None
    if not args.no_fp64:
        a64 = argparse.Namespace(**vars(args))
        a64.steps = max(2, args.steps // 2)
        a64.warmup = max(1, min(args.warmup, 2))
        fp64, _ = time_batch(workloads.c5("fp64", nreals=R, ndomains=args.ndomains), a64, torch, ws, "fp64")
    e2e = None
    if not args.no_e2e and N * R * 8 <= (32 << 30):
        import geosgs

        out = torch.empty(N * R, dtype=torch.float64, pin_memory=True).numpy()
        import ctypes as C

        def e2e_step(i):
            B = geosgs.Batch(probs)
            B.prepare()
            B._check(B.lib.sgs_batch_simulate(B.h, R, None, replica_seed(77 + i), out.ctypes.data_as(C.POINTER(C.c_double))))
            inf = B.info()
            B.close()
            return inf

        e2e_step(0)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        k = max(1, min(3, args.steps))
        infs = [e2e_step(1 + i) for i in range(k)]
        dt = (time.perf_counter() - t0) / k
        e2e = {"value": ws * N * R / dt, "unit": UNIT, "h2d_bytes_per_step": int(infs[-1].h2d_bytes),
               "d2h_bytes_per_step": int(infs[-1].d2h_bytes), "ms_per_step": 1e3 * dt,
               "path": "sgs_batch_create + sgs_batch_prepare + sgs_batch_simulate (FP64 out to pinned host) + "
                       "sgs_batch_destroy"}
    if rank != 0:
        return
    inf = fast["info"]
    sum_m = int(inf.sum_grid_neighbors)
    Rp = (R + 3) // 4 * 4
    # neighbour row reads + value writes (rows of Rp values: 8-byte values in
    # the domains that keep FP64, 4-byte elsewhere), and per grid neighbour an
    # int32 index and a (hi, lo) weight, per node its id, count, CSR row
    # start, (hi, lo) b0 and sigma
    m64, n64 = int(inf.sum_grid_neighbors_fp64), int(fast["nodes_fp64"])
    alg_bytes = (sum_m - m64 + N - n64) * Rp * 4 + (m64 + n64) * Rp * 8 + sum_m * 12 + N * 32
    try:
        peak, peak_src = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["hbm_gbs"]), "measured"
    except Exception:
        peak, peak_src = 6800.0, "fallback"
    ms_sweep = fast["phases"]["sweep"]
    achieved = alg_bytes / (ms_sweep * 1e-3) / 1e9
    cpu = None
    if not args.no_cpu:
        v, cores, sample, _ = cpu_sample_batch(bw, args.cpu_nodes * 4)
        cpu = {"value": v, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample, "extrapolated": True}
    value = ws * N * R / (fast["ms"] * 1e-3)
    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": fast["ms"], "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32 (f64 values)" if inf.values_fp64 else "f32",
        "data": "synthetic (seeded PCG64 domains, variograms, data and paths; on-device Philox normals)",
        "config": batch_config_of(bw, ws),
        "arm": {"precision": "FP32 solve + refinement with exact residuals, FP64 fallback",
                "warm_start": False, "note": "batches run without the learned warm start"},
        "phases_ms": fast["phases"], "nlevels": int(inf.nlevels), "n_prior": int(inf.n_prior),
        "n_fp64_fallback": int(inf.n_fp64_fallback), "bin_systems": [int(x) for x in inf.bin_systems],
        "device_gb": inf.device_bytes / 1e9, "s_create": round(fast["s_create"], 2),
        "values_fp64": int(inf.values_fp64), "weight_l1_max": inf.weight_l1_max,
        "roofline": {"kernel": ("sweep_flow_kernel<float / double, CSR> (one dataflow launch per value precision)"
                                if 0 < n64 < N else
                                "sweep_flow_kernel<%s, CSR> (one dataflow launch)" % ("double" if n64 else "float")),
                     "bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                     "peak_source": peak_src, "traffic": None, "algorithmic_bytes": alg_bytes,
                     "nodes_fp64_values": n64, "ms": ms_sweep},
        "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": int(fast["launches"]) // max(1, args.steps),
        "graph_launches_per_step": fast["graphs"] / max(1, args.steps), "clocks": clk,
        "sweep_config": fast["sweep_config"],
        "sweep_candidates_ms": [round(t["ms"], 3) for t in fast["sweep_tried"]],
    }
    if fp64:
        v64 = ws * N * R / (fp64["ms"] * 1e-3)
        out["fp64_path"] = {"value": v64, "ms_per_step": fp64["ms"], "phases_ms": fp64["phases"]}
        out["speedup_vs_fp64_path"] = value / v64
    print(json.dumps(out))


def main():
    args = parse()
    if args.impl == "reference":
        run_reference(args)
        return
    import torch

    ws, rank, local = dist_setup(args)
    torch.cuda.set_device(local)
    import geosgs
    from geosgs import _build

    _build.build()
    geosgs.load_library()
    try:
        uuid = str(torch.cuda.get_device_properties(local).uuid)
    except Exception:
        uuid = None

    if args.workload == "c5":
        main_batch(args, torch, ws, rank, uuid)
        return
    wl = workload(args.workload, "fp32", args.nreals, args.grid, args.ndata)
    N, R = wl.domain.nelements(), wl.nreals

    # the learned warm start: a network trained on systems the method
    # generates (random 3D variograms, the workload's maxneighbors), before
    # any timed region
    params, training = None, None
    if not args.no_learned:
        from geosgs import learned

        if args.learned_systems is None:
            args.learned_systems = 10_000_000 if args.workload == "c4" else 600_000
        t0 = time.perf_counter()
        feat, count, target = learned.generate(args.learned_systems, seed=11, torch=torch, dims=(48, 48, 32),
                                               k=wl.method.maxneighbors)
        t_gen = time.perf_counter() - t0
        t0 = time.perf_counter()
        params, hist = learned.train(feat, count, target, torch, epochs=args.learned_epochs, batch=16384, lr=3e-3)
        training = {"systems": args.learned_systems, "epochs": args.learned_epochs, "final_mse": hist[-1],
                    "mean_sq_target": float((target ** 2).mean()), "s_generate": round(t_gen, 2),
                    "s_train": round(time.perf_counter() - t0, 2)}
        del feat, count, target
        torch.cuda.empty_cache()

    # every arm is timed on the same steps; the headline arm is the metric's
    # named form (learned + FP32) when the network is trained
    wlh = workload(args.workload, "fp32", args.nreals, args.grid, args.ndata)
    wlh.method.warm_start = params is not None
    clocks = ClockSampler(uuid).start()
    head = time_device(wlh, args, torch, ws, network=params)
    clk = clocks.stop()
    fp32 = time_device(wl, args, torch, ws) if params is not None else None
    fp64 = None
    if not args.no_fp64:
        wl64 = workload(args.workload, "fp64", args.nreals, args.grid, args.ndata)
        fp64 = time_device(wl64, args, torch, ws)

    e2e = None
    if not args.no_e2e:
        e2e_s, e2e_inf, _ = time_e2e(wlh, args, torch, ws, max(1, min(3, args.steps)), sweep=head["sweep_config"],
                                     network=params)
        e2e = {"value": ws * N * R / e2e_s, "unit": UNIT,
               "h2d_bytes_per_step": int(e2e_inf.h2d_bytes), "d2h_bytes_per_step": int(e2e_inf.d2h_bytes),
               "ms_per_step": 1e3 * e2e_s,
               "path": ("sgs_plan_create + " + ("sgs_plan_set_network + " if params is not None else "") +
                        "sgs_plan_prepare + sgs_plan_simulate (FP64 out to pinned host) + sgs_plan_destroy"),
               "calls_ms": getattr(time_e2e, "split_ms", None)}

    if rank != 0:
        return

    # roofline of the sweep (kernel c): algorithmic bytes of one sweep
    inf = head["info"]
    sum_m = int(inf.sum_grid_neighbors)
    sv = 8 if inf.values_fp64 else 4
    # neighbour row reads + value writes, plus the sweep tables: per grid
    # neighbour an int32 index and a (hi, lo) float2 weight, per node its id,
    # neighbour count, (hi, lo) b0 and (hi, lo) sigma
    alg_bytes = (sum_m + N) * R * sv + sum_m * 12 + N * 24
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
        peak, peak_src = float(peaks["hbm_gbs"]), "measured"
    except Exception:
        peak, peak_src = 6800.0, "fallback"
    achieved = alg_bytes / (head["ms_sweep"] * 1e-3) / 1e9
    # DRAM traffic of one sweep from the committed ncu capture of the form
    # this workload times (all launches of one sweep), per node-realization
    traffic, tr = None, {}
    try:
        tr = json.load(open(os.path.join(ROOT, "profiles", "sweep_traffic.json")))
        if tr.get("workload") == wl.name and int(tr.get("nreals", 0)) == R:
            traffic = tr["dram_bytes_per_sweep"]
    except Exception:
        pass
    sc = head["sweep_config"]
    form = {0: "sweep_flow_kernel (dataflow launches%s)" % (
                ", levels %d-%d by per-level launches" % (sc["level_lo"], sc["level_hi"] - 1)
                if sc["level_hi"] > sc["level_lo"] else ""),
            1: "sweep_all_kernel (one cooperative launch)",
            2: ("sweep_levelN_kernel<%d> (one launch per level, %d chunks of 4 realizations per thread)"
                % (sc["lanes_g"], sc["lanes_g"]) if sc["lanes_g"] in (2, 4)
                else "sweep_level_kernel (one launch per level)")}[sc["mode"]]
    roofline = {"kernel": form + ": all launches of one sweep", "bound": "hbm",
                "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "peak_source": peak_src, "traffic": traffic,
                "traffic_measured_on": (tr.get("measured_on") if traffic is not None else None),
                "algorithmic_bytes": alg_bytes,
                "ms": head["ms_sweep"]}

    probes = measure_peaks()
    if e2e is not None and probes.get("host_write_gbs"):
        # the FP64 output crosses the CPU-GPU link: the floor of its transfer
        e2e["host_write_gbs"] = probes["host_write_gbs"]
        e2e["d2h_floor_ms"] = e2e["d2h_bytes_per_step"] / probes["host_write_gbs"] / 1e6
        if probes.get("d2h_copy_gbs"):
            e2e["d2h_copy_gbs"] = probes["d2h_copy_gbs"]

    # the solve (kernel b), bound by the FP32 pipe, on the algorithmic FLOP
    # basis (factorization n^3/3, not the cost of the algorithm run); the FP32
    # count of what runs (L D L' with L^-1 carried in place, two products with
    # L^-1 and its transpose; the residuals are integers) is reported beside it
    sm_mhz = float(peaks.get("sm_max_mhz", 2070.0))
    fp32_nominal = 152 * 128 * 2 * sm_mhz * 1e6 / 1e12
    if probes.get("fp32_tflops"):
        fp32_peak, fp32_src = probes["fp32_tflops"], "measured in this run: independent FFMA chains on every SM"
    else:
        fp32_peak, fp32_src = fp32_nominal, "nominal (SM count x lanes x max clock)"

    def solve_roof(res, steps, peak_, src, kernel, executed=True):
        sz = res["system_sizes"]
        nn = np.arange(sz.size, dtype=np.float64)
        fl = solve_flops(sz, steps)
        tf = fl / (res["ms_solve"] * 1e-3) / 1e12
        out_ = {"kernel": kernel, "achieved": tf, "peak": peak_, "unit": "TFLOP/s", "peak_source": src,
                "frac": tf / peak_ if peak_ else None, "algorithmic_flops": fl,
                "flop_basis": "n(n+1)/2 + n^3/3 + 2n^2 + %d x 4n^2 + 2n per system" % steps,
                "systems": int(sz.sum()), "mean_system_size": float(np.sum(sz * nn) / max(1, sz.sum())),
                "ms": res["ms_solve"]}
        if executed:
            ex = float(np.sum(sz * (2 * nn ** 3 / 3 + 4 * nn ** 2)))
            out_["executed_flops"] = ex
            out_["executed_basis"] = "L D L' with its inverse 2n^3/3 + two solves by products 4n^2, FP32 (integer residuals not counted)"
            out_["executed_tflops"] = ex / (res["ms_solve"] * 1e-3) / 1e12
        return out_

    head_steps = wlh.method.refine_steps + (1 if params is not None else 0)
    solve_roofline = solve_roof(head, head_steps, fp32_peak, fp32_src,
                                "solve_fp32_kernel<NMAX> (+ lag table, the rest of the prediction, FP64 fallbacks): "
                                "one solve phase")
    solve_roofline["nominal_peak"] = fp32_nominal
    solve_roofline["gj_pattern_peak"] = probes.get("gj_pattern_tflops")

    # the search (kernel a) on its algorithmic byte basis: a path-rank read (4 B)
    # per grid candidate examined (earlier path nodes tested by the first
    # ranks, template offsets inside the grid), the FP32 coordinates (16 B) of
    # every datum screened, and the row written (k int32 slots, count and
    # grid count); the candidates are counted by the kernel
    kk = int(inf.maxneighbors)
    s_bytes = (4 * int(inf.search_grid_candidates) + 16 * int(inf.search_data_candidates)
               + N * (4 * kk + 8))
    s_gbs = s_bytes / (head["ms_search"] * 1e-3) / 1e9
    search_roofline = {"kernel": "search_kernel: one search", "bound": "hbm", "achieved": s_gbs, "peak": peak,
                       "unit": "GB/s", "frac": s_gbs / peak, "peak_source": peak_src, "algorithmic_bytes": s_bytes,
                       "grid_candidates": int(inf.search_grid_candidates),
                       "data_candidates": int(inf.search_data_candidates),
                       "basis": "4 B per grid candidate + 16 B per datum screened + (4k + 8) B per node written",
                       "note": "latency bound: the rank gathers hit L2 (profiles/kernels_c3_200x200x50_fp32.md)",
                       "ms": head["ms_search"]}

    cpu = None
    if not args.no_cpu:
        v, cores, sample, _ = cpu_sample(wl, args.cpu_nodes)
        cpu = {"value": v, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample, "extrapolated": True}

    def phases(res, learned=False):
        # with the learned warm start the prediction runs on a second stream
        # beside the dependency levels, and the solve waits for what is left
        return {"search": res["ms_search"],
                ("levels_beside_prediction" if learned else "levels"): res["ms_levels"],
                ("solve_after_prediction" if learned else "solve"): res["ms_solve"],
                "sweep": res["ms_sweep"]}

    value = ws * N * R / (head["ms"] * 1e-3)
    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": head["ms"], "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32 (f64 values)" if inf.values_fp64 else "f32",
        "data": "synthetic (seeded PCG64 grid data and path; on-device Philox normals)",
        "config": config_of(wl, ws),
        "arm": {"form": "learned warm start + FP32" if params is not None else "FP32",
                "precision": "FP32 L D L' + refinement with exact residuals, FP64 L D L' fallback",
                "warm_start": params is not None, "refine_steps": head_steps},
        "phases_ms": phases(head, params is not None),
        "nlevels": int(inf.nlevels), "n_prior": int(inf.n_prior), "n_fp64_fallback": int(inf.n_fp64_fallback),
        "warm_start_accepted": int(inf.n_warm_accepted),
        "values_fp64": int(inf.values_fp64), "weight_l1_max": inf.weight_l1_max,
        "roofline": roofline,
        "solve_roofline": solve_roofline,
        "search_roofline": search_roofline,
        "cpu_baseline": cpu,
        "e2e": e2e,
        "gpu_launches": int(head["launches"]) // max(1, args.steps),
        "clocks": clk,
        "sweep_config": {k: v for k, v in sc.items()},
        "sweep_candidates_ms": [round(t["ms"], 3) for t in head["sweep_tried"]],
    }
    if training:
        out["training"] = training
    if fp32:
        v32 = ws * N * R / (fp32["ms"] * 1e-3)
        out["fp32_path"] = {"value": v32, "ms_per_step": fp32["ms"], "phases_ms": phases(fp32),
                            "solve_roofline": solve_roof(fp32, wl.method.refine_steps, fp32_peak, fp32_src,
                                                         "solve_fp32_kernel<NMAX>: one solve phase")}
    if fp64:
        v64 = ws * N * R / (fp64["ms"] * 1e-3)
        fp64_peak = probes.get("fp64_tflops")
        out["fp64_path"] = {"value": v64, "ms_per_step": fp64["ms"], "phases_ms": phases(fp64),
                            "solve_roofline": solve_roof(fp64, 0, fp64_peak, "measured in this run: independent "
                                                         "DFMA chains on every SM" if fp64_peak else None,
                                                         "solve_kernel<double>: one solve phase",
                                                         executed=False)}
        out["speedup_vs_fp64_path"] = value / v64
        if fp32:
            out["fp32_path"]["speedup_vs_fp64_path"] = out["fp32_path"]["value"] / v64
    print(json.dumps(out))


if __name__ == "__main__":
    main()
