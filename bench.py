#!/usr/bin/env python
"""Benchmark of the HSS ULV solve on one GB300 (or N independent replicas).

Workload (the precision configuration the solve-rate metric is quoted on):
a synthetic HSS matrix, n = 65536 as a perfect binary tree of depth 9 with
leafsize 128 and rank k = 32 (leaf D = randn/sqrt(128) + 4I, orthonormal U, V,
R, W, B = 0.5 randn/sqrt(32), seed 3), and r = 32 right-hand sides ~ N(0,1).

One step = one ``hssA \\ B``: ULV factorization + solve, in the mixed form
(FP32 factorization and solve, FP64 HSS-product residual and update, refined
to a relative residual of 1e-10).  The plain FP64 form of the same step is
timed on the same GPU for comparison.  ``value`` counts steps (solves with 32
right-hand sides each) per second over all ranks, with the generators and B
resident in HBM; ``e2e`` is the same step through the C ABI's host-buffer
entry point (``hss_ulvfactsolve_host``) from pinned memory, copies included.
L2 is flushed (a 512 MB write) before every timed step.

``--impl reference`` times the CPU restatement of the reference algorithm
(``oracle/``, NumPy + LAPACK, all host threads) on the same workload.
"""
from __future__ import annotations

import argparse
import gc
import ctypes
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "HSS ULV solves/s + p50/p99 at 1e-10 resid (mixed+batched vs plain FP64 GPU)"
UNIT = "solves/s"


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=200)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--n", type=int, default=65536)
    p.add_argument("--leafsize", type=int, default=128)
    p.add_argument("--rank", type=int, default=32)
    p.add_argument("--rhs", type=int, default=32)
    p.add_argument("--tol", type=float, default=1e-10)
    p.add_argument("--seed", type=int, default=3)
    p.add_argument("--roofline-kernel", default="factor_leaf")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-extras", action="store_true",
                   help="precision workload: skip the batching and compression headlines")
    p.add_argument("--workload", default="precision",
                   choices=["precision", "serve", "batch", "compress", "matvec", "steps"])
    p.add_argument("--compress-n", type=int, default=16384)
    p.add_argument("--requests", type=int, default=10000)
    p.add_argument("--rate", type=float, default=500.0)
    p.add_argument("--rates", default="500,1000,2000,4000,8000", help="offered loads of the serving sweep (requests/s)")
    p.add_argument("--pool", type=int, default=32)
    p.add_argument("--budget-gb", type=float, default=120.0)
    p.add_argument("--matrices", type=int, default=256)
    return p.parse_args()


def config(args, n_gpus):
    return {
        "workload": (f"precision: synthetic HSS n={args.n}, perfect tree leafsize {args.leafsize}, "
                     f"k={args.rank}, r={args.rhs} RHS; step = ULV factor + solve (hssA\\B), "
                     f"FP32 ULV + FP64-residual refinement to {args.tol:g}"),
        "n": args.n, "leafsize": args.leafsize, "k": args.rank, "rhs": args.rhs, "tol": args.tol,
        "seed": args.seed, "l2": "flushed before every timed step (512 MB write)",
        "parallelism": "replicas" if n_gpus > 1 else "single",
        "launch": ("dedicated stream; every step one replayed CUDA graph (factorization, solve and the "
                   "refinement loop, whose convergence check runs on the device as the condition of a graph "
                   "while node); step = hss_ulvfactsolve (first solve pipelined behind the factorization); "
                   "solve kernels autotuned per level in setup"),
    }


# ---------------------------------------------------------------------------
# CPU side: the oracle restatement (reference arm and cpu_baseline)
# ---------------------------------------------------------------------------


def cpu_solve_sample(args, calls):
    import numpy as np
    from oracle import hss_oracle as orc
    h = orc.synthetic_hss(args.n, args.leafsize, args.rank, np.random.default_rng(args.seed))
    b = np.random.default_rng(1).standard_normal((args.n, args.rhs))
    times = []
    for _ in range(calls):
        t0 = time.perf_counter()
        orc.ulvfactsolve(h, b)
        times.append(time.perf_counter() - t0)
    return times


def max_over_ranks(value, device):
    """The largest of `value` over the ranks of the default process group: a
    one-element all-reduce on `device` ("cuda" under NCCL, "cpu" under gloo).
    Every rank times its own replica; the job's time is the slowest rank's."""
    import torch
    import torch.distributed as td
    t = torch.tensor([float(value)], dtype=torch.float64, device=device)
    td.all_reduce(t, op=td.ReduceOp.MAX)
    return float(t.item())


def job_rate(world, steps_per_rank, seconds):
    """Whole-job throughput of `world` independent replicas that each ran
    `steps_per_rank` steps in at most `seconds` (the max over ranks)."""
    return world * steps_per_rank / seconds


def run_reference(args, rank, world):
    if rank != 0:
        return 0
    for _ in range(args.warmup):
        cpu_solve_sample(args, 1)
    times = cpu_solve_sample(args, args.steps)
    ms = 1000.0 * statistics.mean(times)
    value = 1000.0 / ms
    cores = os.cpu_count()
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "impl": "reference", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": config(args, world),
        "p50_ms": 1000.0 * statistics.median(times),
        "p99_ms": 1000.0 * sorted(times)[min(len(times) - 1, int(math.ceil(0.99 * len(times))) - 1)],
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{args.steps} full hssA\\B calls (n={args.n}, r={args.rhs}) with the "
                                   "NumPy/LAPACK restatement of ulvfactsolve (Julia is not installed)"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------


class Clocks:
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=self.fh, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.fh.close()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in open(self.path):
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None, "reasons": sorted(reasons),
                "samples": len(sm)}


# ---------------------------------------------------------------------------
# GPU arm
# ---------------------------------------------------------------------------


# DRAM bytes (read + write) of one leaf-level launch of ulv_factor_blk_kernel<float, 128>
# on the default workload (n = 65536, leafsize 128, k = 32), from one ncu capture
# of that launch (dram__bytes_read.sum + dram__bytes_write.sum).  It belongs to
# that kernel and size only; re-capture it when the kernel changes.
FACTOR_LEAF_TRAFFIC = {(65536, 128, 32): 142420992}
# the same for one r = 1 launch of pmv_flat_kernel (FP64 product) on that tree
MATVEC_R1_TRAFFIC = {(65536, 128, 32): 130451968}


def factor_leaf_bytes(A, factor_itemsize):
    """Algorithmic bytes of one leaf-level ULV launch: read every leaf's D, U, V
    (FP64 generators) once and write its reduced blocks + tau vectors once."""
    tot_read = tot_write = 0

    def walk(x, root):
        nonlocal tot_read, tot_write
        if x.leafnode:
            m, n = x.D.shape
            ku, kv = (0, 0) if root else (x.U.shape[1], x.V.shape[1])
            tot_read += 8 * (m * n + m * ku + n * kv)
            k = min(ku, m)
            tot_write += factor_itemsize * (m * n + m * ku + n * kv + k + (m - k))
            return
        walk(x.A11, False)
        walk(x.A22, False)

    walk(A, True)
    return tot_read + tot_write


def run_ours(args, rank, world, local_rank):
    import numpy as np
    import torch
    import __graft_entry__ as g

    torch.cuda.set_device(local_rank)
    pkg = g.load_package()
    from hssmatrices_gb300 import linalg as L
    dist = world > 1
    if dist:
        import torch.distributed as td

    def barrier():
        if dist:
            td.barrier()
        torch.cuda.synchronize()

    n, r = args.n, args.rhs
    A = pkg.synthetic_hss(n, args.leafsize, args.rank, np.random.default_rng(args.seed))
    dev = A.device()
    # a dedicated stream, so that the library replays each step's per-level
    # launch sequences as CUDA graphs (HSS_OPT_GRAPHS; no capture on the
    # legacy default stream)
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    assert dev.lib.hss_set_option(4, 1) == 0
    rng = np.random.default_rng(1)
    Bh = rng.standard_normal((n, r))
    # an n x r column-major matrix is an r x n row-major tensor
    dB = torch.from_numpy(np.ascontiguousarray(Bh.T)).cuda()
    dX = torch.zeros_like(dB)
    flush = torch.empty(512 * 1024 * 1024, dtype=torch.uint8, device="cuda")
    F32 = dev.ulvfactor("fp32", stream=stream)
    F64 = dev.ulvfactor("fp64", stream=stream)
    # per-level solve kernels and residual product chosen by the library's
    # autotuner on scratch right-hand sides (setup, outside the timed region)
    F32.autotune(r, stream=stream)
    F64.autotune(r, stream=stream)

    # one step: factorization + solve in one call (hss_ulvfactsolve: the first
    # solve's upward sweep runs one level behind the factorization)
    def step32():
        return F32.factsolve_device(dB, n, r, dX, n, tol=args.tol, maxit=20, stream=stream)

    def step64(dX64):
        return F64.factsolve_device(dB, n, r, dX64, n, tol=0.0, stream=stream)

    for _ in range(args.warmup):
        step32()
    barrier()
    # timed region: K mixed-precision steps
    clocks = Clocks(local_rank)
    clocks.start()
    launches0 = L.launch_counter()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(args.steps)]
    iters = []
    barrier()
    for i in range(args.steps):
        flush.zero_()
        ev[i][0].record(stream)
        st = step32()
        ev[i][1].record(stream)
        iters.append(st.iterations)
    barrier()
    launches = L.launch_counter() - launches0
    times = [a.elapsed_time(b) for a, b in ev]
    total_ms = sum(times)
    # the dominant kernel's launch duration: CUDA events around each of its
    # launches over a second run of K steps (event bracketing replaces the
    # graph replay by the same launches issued one by one)
    L.trace_begin(args.roofline_kernel)
    for i in range(args.steps):
        flush.zero_()
        step32()
    barrier()
    k_ms, k_cnt = L.trace_end()
    clk = clocks.stop()
    # per kernel kind: device time per mixed step (CUDA events around each
    # launch of one kind at a time, a few extra steps per kind)
    breakdown = {}
    for kind in ("factor_leaf", "factor_merge", "solve_up", "solve_down", "mv_dx", "mv_leaf", "mv_up", "mv_down",
                 "mv_final"):
        L.trace_begin(kind)
        for _ in range(3):
            step32()
        kms, _kn = L.trace_end()
        breakdown[kind] = kms / 3
    if dist:
        total_ms = max_over_ranks(total_ms, "cuda")
    ms = total_ms / args.steps
    value = job_rate(world, args.steps, total_ms / 1000.0)
    Xh = dX.cpu().numpy().T
    res32 = float(np.max(np.linalg.norm(Bh - pkg.matmul(A, Xh), axis=0) / np.linalg.norm(Bh, axis=0)))
    # plain FP64 form on the same GPU
    dX64 = torch.zeros_like(dB)
    for _ in range(max(1, args.warmup)):
        step64(dX64)
    ev64 = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
            for _ in range(args.steps)]
    barrier()
    for i in range(args.steps):
        flush.zero_()
        ev64[i][0].record(stream)
        step64(dX64)
        ev64[i][1].record(stream)
    barrier()
    t64 = [a.elapsed_time(b) for a, b in ev64]
    ms64 = sum(t64) / args.steps
    breakdown64 = {}
    for kind in ("factor_leaf", "factor_merge", "solve_up", "solve_down"):
        L.trace_begin(kind)
        step64(dX64)
        kms, _kn = L.trace_end()
        breakdown64[kind] = kms
    X64 = dX64.cpu().numpy().T
    res64 = float(np.max(np.linalg.norm(Bh - pkg.matmul(A, X64), axis=0) / np.linalg.norm(Bh, axis=0)))
    # end to end through the host-buffer C entry point, pinned memory
    import ctypes as C
    Bp = torch.from_numpy(np.asfortranarray(Bh).T.copy()).pin_memory()   # r x n rows = columns of B
    Xp = torch.zeros_like(Bp).pin_memory()
    stats = pkg._lib.SolveStats()
    lib = dev.lib

    def e2e_call():
        rc = lib.hss_ulvfactsolve_host(dev.handle, pkg._lib.HSS_PREC_FP32,
                                       C.cast(C.c_void_p(Bp.data_ptr()), pkg._lib.PD), n, r,
                                       C.cast(C.c_void_p(Xp.data_ptr()), pkg._lib.PD), n, args.tol, 20, C.byref(stats))
        pkg._lib.check(rc)

    for _ in range(args.warmup):
        e2e_call()
    barrier()
    e2e_t = []
    for _ in range(args.steps):
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        e2e_call()
        e2e_t.append(time.perf_counter() - t0)
    barrier()
    e2e_total = sum(e2e_t)
    if dist:
        e2e_total = max_over_ranks(e2e_total, "cuda")
    e2e_value = job_rate(world, args.steps, e2e_total)
    # the HSS x dense product (FP64 hss_matmul, persistent kernel) on the same
    # tree: r = 1 and r = rhs columns, L2 flushed before each call
    matvec_us = {}
    for rr in sorted({1, r}):
        mB = torch.randn((rr, n), dtype=torch.float64, device="cuda")
        mC = torch.empty_like(mB)
        for _ in range(3):
            dev.matmul_device(mB, n, rr, mC, n, stream=stream)
        ev_m = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(20)]
        torch.cuda.synchronize()
        for a, b in ev_m:
            flush.zero_()
            a.record(stream)
            dev.matmul_device(mB, n, rr, mC, n, stream=stream)
            b.record(stream)
        torch.cuda.synchronize()
        matvec_us[rr] = 1000.0 * statistics.median(a.elapsed_time(b) for a, b in ev_m)
        del mB, mC
    if rank != 0:
        return 0
    # roofline of the dominant kernel (per launch)
    per_launch_ms = k_ms / max(k_cnt, 1)
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
        peak, peak_src = float(peaks["hbm_gbs"]), "measured"
    except Exception:
        peak, peak_src = 6800.0, "fallback"
    alg_bytes = factor_leaf_bytes(A, 4) if args.roofline_kernel == "factor_leaf" else None
    achieved = alg_bytes / (per_launch_ms * 1e-3) / 1e9 if alg_bytes and per_launch_ms > 0 else None
    traffic = (FACTOR_LEAF_TRAFFIC.get((n, args.leafsize, args.rank)) if args.roofline_kernel == "factor_leaf"
               else None)
    roof = {"kernel": args.roofline_kernel, "bound": "hbm", "achieved": achieved, "peak": peak,
            "unit": "GB/s", "frac": (achieved / peak) if achieved else None, "traffic": traffic,
            "traffic_source": "ncu capture of one leaf-level launch at this size" if traffic else None,
            "peak_source": peak_src, "launch_ms": per_launch_ms, "launches": k_cnt,
            "launch_timing": "CUDA events around every launch of the kernel over a second run of the K steps "
                             "(launches issued one by one instead of replayed as a graph)",
            "algorithmic_bytes": alg_bytes}
    cpu = None
    if not args.no_cpu_baseline:
        ct = cpu_solve_sample(args, 2)
        cms = 1000.0 * min(ct)
        cpu = {"value": 1000.0 / cms, "unit": UNIT, "cores": os.cpu_count(), "kind": "port",
               "sample": f"2 full hssA\\B calls (n={n}, r={r}), NumPy/LAPACK restatement, best of 2"}
    st_sorted = sorted(times)
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "fp32+fp64", "data": "synthetic", "config": config(args, world),
        "p50_ms": statistics.median(times),
        "p99_ms": st_sorted[min(len(st_sorted) - 1, int(math.ceil(0.99 * len(st_sorted))) - 1)],
        "rhs_per_s": value * r, "refine_iters": iters, "residual": res32,
        "fp64": {"solves_per_s": world * 1000.0 / ms64, "ms_per_step": ms64, "residual": res64,
                 "p50_ms": statistics.median(t64), "breakdown_ms_per_step": breakdown64},
        "speedup_vs_fp64": ms64 / ms,
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": 8 * n * r,
                "d2h_bytes_per_step": 8 * n * r, "ms_per_step": 1000.0 * e2e_total / args.steps},
        "roofline": roof, "cpu_baseline": cpu, "clocks": clk, "gpu_launches": launches,
        "breakdown_ms_per_step": breakdown,
        "factor_bytes": {"fp32": F32.nbytes(), "fp64": F64.nbytes()},
        "autotune": {"fp32": F32.tuning(), "fp64": F64.tuning()},
    }
    for rr, us in matvec_us.items():
        line[f"matvec_r{rr}_us"] = us
    # the batching and compression workloads' headlines (their own runs,
    # --workload batch / compress, add the FP64 and CPU comparisons)
    if not args.no_extras:
        del F32, F64, dev
        gc.collect()
        torch.cuda.empty_cache()
        line["batch"] = batch_headline(pkg, args)
        line["batch_ms"] = line["batch"]["ms_per_step"]
        gc.collect()
        torch.cuda.empty_cache()
        line["compress"] = compress_headline(pkg, args.compress_n)
        line["compress_ms"] = line["compress"]["ms"]
    print(json.dumps(line), flush=True)
    return 0


# ---------------------------------------------------------------------------
# serving workload (Poisson request stream) and batched workload
# ---------------------------------------------------------------------------


def _pct(v, q):
    v = sorted(v)
    return v[min(len(v) - 1, max(0, int(math.ceil(q * len(v))) - 1))]


def _serve_once(pkg, serve, args, rate, precision, overlap=True, check=True):
    """One replay of the request stream at `rate` requests/s; returns its summary."""
    import torch
    reqs, _pool = serve.synthetic_requests(n_requests=args.requests, seed=3, rate=rate, pool_size=args.pool)
    torch.cuda.synchronize()
    srv = serve.HssServer(budget_bytes=int(args.budget_gb * 1e9), precision=precision, tol=args.tol,
                          overlap=overlap)
    t0 = time.perf_counter()
    done = serve.run_stream(srv, reqs)
    makespan = time.perf_counter() - t0
    lat = [1000.0 * (r.done - r.arrival) for r in done]
    slat = [1000.0 * (r.done - r.arrival) for r in done if r.kind == "solve"]
    flat = [1000.0 * (r.done - r.arrival) for r in done if r.kind == "factor"]
    nsolve = sum(1 for r in done if r.kind == "solve")
    nrhs = sum(r.rhs.shape[0] for r in done if r.kind == "solve")
    out = {"offered_per_s": rate, "precision": precision, "overlap": overlap,
           "solves_per_s": nsolve / makespan, "requests_per_s": len(done) / makespan, "rhs_per_s": nrhs / makespan,
           "p50_ms": _pct(lat, 0.5), "p99_ms": _pct(lat, 0.99), "solve_p50_ms": _pct(slat, 0.5),
           "solve_p99_ms": _pct(slat, 0.99), "factor_p50_ms": _pct(flat, 0.5), "factor_p99_ms": _pct(flat, 0.99),
           "makespan_s": makespan, "arrival_span_s": reqs[-1].arrival, "factor_batches": srv.factor_batches,
           "solve_batches": srv.solve_batches, "overlapped_factor_batches": srv.overlapped,
           "evictions": srv.evictions, "reloads": srv.reloads}
    if check:
        # the true residual of every served solve (FP64 product on the GPU)
        worst, checked = 0.0, 0
        by_matrix = {}
        for q in done:
            if q.kind == "solve":
                by_matrix.setdefault(q.matrix, []).append(q)
        for mi, lst in by_matrix.items():
            dv = pkg.linalg.DeviceHss(pkg.HssMatrix.from_tree(srv.matrices[mi]))
            for q in lst:
                R = q.rhs.clone()
                dv.matmul_device(q.out, dv.n, q.rhs.shape[0], R, dv.m, alpha=-1.0, beta=1.0)
                worst = max(worst, float((torch.linalg.norm(R, dim=1) / torch.linalg.norm(q.rhs, dim=1)).max()))
                checked += 1
            del dv
        out["max_residual"] = worst
        out["residuals_checked"] = checked
    out["resident_gb_at_end"] = srv.used / 1e9
    srv.resident.clear()
    del srv, done, reqs
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return out


def run_serve(args):
    """Serving: Poisson streams of factor (20%) and solve (80%) requests at rising
    offered loads; the continuous-batching server (factor and solve batches on two
    streams, overlapping) in FP32 + refinement and in plain FP64 through the same
    batcher, plus the FP32 server without overlap at the highest load."""
    import torch
    import __graft_entry__ as g
    pkg = g.load_package()
    from hssmatrices_gb300 import serve
    rates = [float(x) for x in args.rates.split(",")]
    # warm-up: both precisions, a short stream
    for prec in ("fp32", "fp64"):
        w = serve.HssServer(budget_bytes=int(args.budget_gb * 1e9), precision=prec, tol=args.tol)
        reqs, _ = serve.synthetic_requests(n_requests=40, seed=9, rate=4000.0, pool_size=4, n_range=(2048, 8192))
        serve.run_stream(w, reqs)
        del w, reqs
    torch.cuda.synchronize()
    clocks = Clocks(0)
    clocks.start()
    sweep32 = [_serve_once(pkg, serve, args, rate, "fp32") for rate in rates]
    clk = clocks.stop()
    sweep64 = [_serve_once(pkg, serve, args, rate, "fp64", check=False) for rate in rates]
    no_overlap = _serve_once(pkg, serve, args, rates[-1], "fp32", overlap=False, check=False)
    best = max(sweep32, key=lambda x: x["solves_per_s"])
    head = sweep32[rates.index(args.rate)] if args.rate in rates else best
    line = {
        "metric": METRIC, "value": best["solves_per_s"], "unit": UNIT, "n_gpus": 1, "steps": args.requests,
        "warmup": 1, "ms_per_step": 1000.0 * best["makespan_s"] / args.requests, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "fp32+fp64", "data": "synthetic",
        "config": {"workload": (f"serving: {args.requests} Poisson requests per run (seed 3) at offered loads "
                                f"{rates} per s, 20% factor (n log-uniform 2048..65536, k 16..48, leafsize 128, "
                                f"pool of {args.pool} matrices), 80% solve (r 1..32) against resident "
                                f"factorizations; {args.budget_gb:g} GB HBM budget; value = the highest "
                                f"served solves/s over the loads (FP32 + refinement)"),
                   "tol": args.tol},
        "p50_ms": head["p50_ms"], "p99_ms": head["p99_ms"], "at_offered_per_s": head["offered_per_s"],
        "max_residual": max(x["max_residual"] for x in sweep32),
        "residuals_checked": sum(x["residuals_checked"] for x in sweep32),
        "sweep_fp32": sweep32, "sweep_fp64_same_batcher": sweep64, "fp32_without_overlap": no_overlap,
        "clocks": clk,
    }
    print(json.dumps(line), flush=True)
    return 0


def batch_trees(pkg, count):
    """The batching workload's matrices (seed 2): n uniform 1024..16384 step 128,
    leafsize in {64, 128, 256}, k 8..48, and r 1..16 right-hand sides each."""
    import numpy as np
    rng = np.random.default_rng(2)
    trees, rs = [], []
    for _ in range(count):
        n = int(rng.integers(1024 // 128, 16384 // 128 + 1)) * 128
        ls = int(rng.choice([64, 128, 256]))
        k = int(rng.integers(8, 49))
        trees.append(pkg.synthetic_hss(n, ls, k, rng))
        rs.append(int(rng.integers(1, 17)))
    return trees, rs


def batch_headline(pkg, args, steps=5):
    """The batching workload's headline alone: FP32 ULV factor + solve with
    refinement of all matrices of the forest per step (graphs, autotuned), the
    mean of `steps` timed steps, and the largest true residual."""
    import torch
    trees, rs = batch_trees(pkg, args.matrices)
    forest = pkg.DeviceHss.from_trees(trees)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        Bs = [torch.randn((r, t.size()[0]), dtype=torch.float64, device="cuda") for t, r in zip(trees, rs)]
        Xs = [torch.empty_like(b) for b in Bs]
    stream.synchronize()
    ns = [t.size()[0] for t in trees]
    F = forest.ulvfactor("fp32", stream=stream)
    F.autotune(max(rs), stream=stream)
    for _ in range(3):
        F.refactor(stream=stream)
        F.solve_batch_device(Bs, ns, rs, Xs, ns, tol=args.tol, maxit=20, stream=stream)
    stream.synchronize()
    times = []
    for _ in range(steps):
        stream.synchronize()
        t0 = time.perf_counter()
        F.refactor(stream=stream)
        F.solve_batch_device(Bs, ns, rs, Xs, ns, tol=args.tol, maxit=20, stream=stream)
        stream.synchronize()
        times.append(time.perf_counter() - t0)
    with torch.cuda.stream(stream):
        Rs = [b.clone() for b in Bs]
        forest.matmul_batch_device(Xs, ns, rs, Rs, ns, alpha=-1.0, beta=1.0, stream=stream)
        res = max(float((torch.linalg.norm(R, dim=1) / torch.linalg.norm(b, dim=1)).max()) for R, b in zip(Rs, Bs))
    stream.synchronize()
    ms = 1000.0 * statistics.mean(times)
    return {"workload": f"{args.matrices} matrices (the batch workload), FP32 ULV factor + solve to {args.tol:g}",
            "ms_per_step": ms, "matrix_solves_per_s": 1000.0 * args.matrices / ms, "max_residual": res,
            "steps": steps}


def compress_headline(pkg, n, steps=3):
    """The compression workload's headline alone: randcompress_adaptive of the
    Cauchy matrix (n, leafsize 128, kest 10, 1e-9) with FP64 sampling, median
    of `steps` calls."""
    import numpy as np
    import torch
    from hssmatrices_gb300 import compression as CP
    Ad = CP.DenseDevice.__new__(CP.DenseDevice)
    Ad.t, Ad.m, Ad.n, Ad.lda = cauchy_device(n), n, n, n
    cl = pkg.bisection_cluster(n, 128)

    def compress():
        return pkg.randcompress_adaptive(Ad, cl, cl, kest=10, atol=1e-9, rtol=1e-9, noversampling=10, stepsize=20,
                                         rng=np.random.default_rng(1), device=True)

    compress()
    torch.cuda.synchronize()
    times = []
    for _ in range(steps):
        t0 = time.perf_counter()
        compress()
        torch.cuda.synchronize()
        times.append(time.perf_counter() - t0)
    del Ad
    torch.cuda.empty_cache()
    return {"workload": f"randcompress_adaptive, Cauchy matrix n = {n} (the compress workload)",
            "ms": 1000.0 * statistics.median(times), "steps": steps}


def run_batch(args):
    """Batching: many independent HSS matrices of uneven sizes, leaf sizes and ranks
    in one forest, factored and solved with one launch per tree level; FP64 and
    FP32+refinement vs looping plain FP64 per matrix."""
    import numpy as np
    import torch
    import __graft_entry__ as g
    pkg = g.load_package()
    trees, rs = batch_trees(pkg, args.matrices)
    forest = pkg.DeviceHss.from_trees(trees)
    stream = torch.cuda.Stream()   # graphs need a non-default stream
    with torch.cuda.stream(stream):
        Bs = [torch.randn((r, t.size()[0]), dtype=torch.float64, device="cuda") for t, r in zip(trees, rs)]
        Xs = [torch.empty_like(b) for b in Bs]
    stream.synchronize()
    ns = [t.size()[0] for t in trees]
    lib = forest.lib
    assert lib.hss_set_option(4, 1) == 0   # HSS_OPT_GRAPHS: factor and solve launch sequences as CUDA graphs
    out = {}
    tuning = None
    for prec, tol in (("fp64", 0.0), ("fp32", args.tol)):
        F = forest.ulvfactor(prec, stream=stream)
        if prec == "fp32":
            tuning = F.autotune(max(rs), stream=stream)   # per-level kernel choice, timed once
        for _ in range(max(2, args.warmup)):   # the second identical call is captured
            F.refactor(stream=stream)
            F.solve_batch_device(Bs, ns, rs, Xs, ns, tol=tol, maxit=20, stream=stream)
        stream.synchronize()
        times = []
        for _ in range(args.steps):
            stream.synchronize()
            t0 = time.perf_counter()
            F.refactor(stream=stream)
            F.solve_batch_device(Bs, ns, rs, Xs, ns, tol=tol, maxit=20, stream=stream)
            stream.synchronize()
            times.append(time.perf_counter() - t0)
        # true residual of every matrix: R = B - A X with the FP64 product of the forest
        with torch.cuda.stream(stream):
            Rs = [b.clone() for b in Bs]
            forest.matmul_batch_device(Xs, ns, rs, Rs, ns, alpha=-1.0, beta=1.0, stream=stream)
            res = max(float((torch.linalg.norm(R, dim=1) / torch.linalg.norm(b, dim=1)).max())
                      for R, b in zip(Rs, Bs))
        stream.synchronize()
        out[prec] = {"ms_per_step": 1000.0 * statistics.mean(times), "p50_ms": 1000.0 * statistics.median(times),
                     "max_residual": res}
        del F, Rs
    lib.hss_set_option(4, 0)
    # looping plain FP64 per matrix (separate plans, one matrix at a time)
    devs = [pkg.linalg.DeviceHss(t) for t in trees]
    facs = [d.ulvfactor("fp64") for d in devs]
    torch.cuda.synchronize()
    times = []
    for _ in range(max(1, min(args.steps, 3))):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for d, f, b, x, r in zip(devs, facs, Bs, Xs, rs):
            f.refactor()
            f.solve_device(b, d.n, r, x, d.n, tol=0.0)
        torch.cuda.synchronize()
        times.append(time.perf_counter() - t0)
    loop_ms = 1000.0 * statistics.mean(times)
    m32 = out["fp32"]["ms_per_step"]
    line = {
        "metric": METRIC, "value": 1000.0 * args.matrices / m32, "unit": "matrix solves/s", "n_gpus": 1,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": m32, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "fp32+fp64", "data": "synthetic",
        "config": {"workload": (f"batching: {args.matrices} matrices, n uniform 1024..16384 step 128 (seed 2), "
                                f"leafsize in {{64,128,256}}, k 8..48, r 1..16; step = factor + solve of all, "
                                f"FP32 ULV + refinement to {args.tol:g}; one forest plan, one launch per tree "
                                f"level across all matrices, factor/solve sequences replayed as CUDA graphs, "
                                f"solve kernels autotuned per level")},
        "autotune": tuning,
        "max_residual_all_matrices": out["fp32"]["max_residual"],
        "fp64_batched_ms": out["fp64"]["ms_per_step"], "fp64_batched_max_residual": out["fp64"]["max_residual"],
        "fp64_loop_ms": loop_ms,
        "speedup_vs_fp64_loop": loop_ms / m32, "total_rhs": sum(rs),
    }
    print(json.dumps(line), flush=True)
    return 0


def cauchy_device(n):
    """A_ij = 1/(x_i - x_j), 1 on the diagonal, x = n uniform points in [-1, 1], built
    on the device as its column-major storage (the (n, n) row-major tensor of A^T)."""
    import torch
    x = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda")
    t = x[None, :] - x[:, None]          # t[j, i] = x_i - x_j = A_ij
    t.reciprocal_()
    t.diagonal().fill_(1.0)
    return t


def run_compress(args):
    """Config 2: randcompress_adaptive of the Cauchy kernel matrix (n = 16384,
    leafsize 128, kest 10, atol = rtol = 1e-9, noversampling 10, stepsize 20),
    then a 64-RHS product and a 64-RHS FP64 ULV factor + solve of the result."""
    import numpy as np
    import torch
    import __graft_entry__ as g
    pkg = g.load_package()
    from hssmatrices_gb300 import compression as CP
    n = args.compress_n
    tol = 1e-9
    Ad = CP.DenseDevice.__new__(CP.DenseDevice)
    Ad.t, Ad.m, Ad.n, Ad.lda = cauchy_device(n), n, n, n
    cl = pkg.bisection_cluster(n, 128)
    flops_per_col = 2.0 * n * n

    def compress(stats=None, prec="fp64"):
        return pkg.randcompress_adaptive(Ad, cl, cl, kest=10, atol=tol, rtol=tol, noversampling=10, stepsize=20,
                                         rng=np.random.default_rng(1), stats=stats, device=True,
                                         sample_precision=prec)

    for _ in range(max(1, args.warmup)):
        dev = compress()
    torch.cuda.synchronize()
    # sample-product kernel alone: A * Omega with 20 columns (one test round's product)
    Om = torch.randn((20, n), dtype=torch.float64, device="cuda")
    out = torch.empty_like(Om)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ts = []
    for _ in range(5):
        e0.record()
        CP.sample(Ad, Om, out=out)
        e1.record()
        torch.cuda.synchronize()
        ts.append(e0.elapsed_time(e1))
    gemm_ms = statistics.median(ts)
    # the same product in double-float arithmetic (the mixed-precision form)
    ref20 = out.clone()
    with CP._SamplePrecision(Ad, "df"):
        ts = []
        for _ in range(5):
            e0.record()
            CP.sample(Ad, Om, out=out)
            e1.record()
            torch.cuda.synchronize()
            ts.append(e0.elapsed_time(e1))
    gemm_df_ms = statistics.median(ts)
    gemm_df_err = float(torch.linalg.norm(out - ref20) / torch.linalg.norm(ref20))
    clocks = Clocks(0)
    clocks.start()
    times = []
    st = {}
    for _ in range(args.steps):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        dev = compress(st)
        torch.cuda.synchronize()
        times.append(time.perf_counter() - t0)
    ck = clocks.stop()
    ms = 1000.0 * statistics.median(times)
    # mixed form: double-float sample products, FP64 rank decisions
    st_df = {}
    dev_df = compress(st_df, "df")
    times_df = []
    for _ in range(min(args.steps, 50)):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        dev_df = compress(st_df, "df")
        torch.cuda.synchronize()
        times_df.append(time.perf_counter() - t0)
    ms_df = 1000.0 * statistics.median(times_df)
    h = dev.to_host()
    # the compressed matrix on the hot path: 64-RHS product and FP64 ULV solve
    rng = np.random.default_rng(1)
    Bh = rng.standard_normal((n, 64))
    dB = torch.from_numpy(np.ascontiguousarray(Bh.T)).cuda()
    dC = torch.empty_like(dB)
    dev.matmul_device(dB, n, 64, dC, n)
    F = dev.ulvfactor("fp64")
    dX = torch.empty_like(dB)
    F.solve_device(dB, n, 64, dX, n, tol=0.0)
    torch.cuda.synchronize()
    tm, tf = [], []
    for _ in range(5):
        t0 = time.perf_counter()
        dev.matmul_device(dB, n, 64, dC, n)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        F.refactor()
        F.solve_device(dB, n, 64, dX, n, tol=0.0)
        torch.cuda.synchronize()
        tm.append(t1 - t0)
        tf.append(time.perf_counter() - t1)
    # accuracy against the dense matrix (on the device)
    At = Ad.t   # column-major A
    AX = (dX @ At)                      # (64, n) row-major = columns of A X
    solve_res = float(torch.linalg.norm(AX - dB) / torch.linalg.norm(dB))
    Ay = (dB @ At)
    mv_err = float(torch.linalg.norm(dC - Ay) / torch.linalg.norm(Ay))
    dev_df.matmul_device(dB, n, 64, dC, n)
    mv_err_df = float(torch.linalg.norm(dC - Ay) / torch.linalg.norm(Ay))
    samples = st.get("samples", 0)
    cols = 2 * samples + 2 * 20 * st.get("rounds", 0)   # initial samples + every test round
    line = {
        "metric": "randcompress_adaptive compressions/s (config 2)", "value": 1000.0 / ms,
        "unit": "compressions/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": (f"compress: Cauchy kernel 1/(x_i-x_j) on {n} points in [-1,1], dense FP64 "
                                f"resident; bisection_cluster leafsize 128; randcompress_adaptive kest 10, "
                                f"atol=rtol=1e-9, noversampling 10, stepsize 20, Omega from default_rng(1)")},
        "rounds": st.get("rounds"), "k": st.get("k"), "hssrank": int(pkg.hssrank(h)),
        "sample_gemm": {"ms_20cols": gemm_ms, "tflops": flops_per_col * 20 / (gemm_ms * 1e-3) / 1e12,
                        "fp64_peak_tflops_measured": 1.204},
        "sample_columns_per_compression": cols,
        "mixed_df_sampling": {
            "ms_per_compression": ms_df, "compressions_per_s": 1000.0 / ms_df, "speedup_vs_fp64": ms / ms_df,
            "rounds": st_df.get("rounds"), "k": st_df.get("k"), "hssrank": int(pkg.hssrank(dev_df.to_host())),
            "matvec_rel_err_vs_dense": mv_err_df,
            "sample_gemm_ms_20cols": gemm_df_ms, "sample_gemm_rel_diff_vs_fp64": gemm_df_err,
            "sample_gemm_fp64_equiv_tflops": flops_per_col * 20 / (gemm_df_ms * 1e-3) / 1e12},
        "matvec64_ms": 1000.0 * statistics.median(tm), "matvec_rel_err_vs_dense": mv_err,
        "ulv64_fp64_ms": 1000.0 * statistics.median(tf), "ulv_rel_residual_vs_dense": solve_res,
        "clocks": ck,
    }
    if not args.no_cpu_baseline:
        from oracle import hss_oracle as orc
        A = orc.cauchy_matrix(n)
        ocl = orc.bisection_cluster(n, 128)
        t0 = time.perf_counter()
        orc.randcompress_adaptive(A, ocl, ocl, 10, tol, tol, 10, 20, rng=np.random.default_rng(1))
        dt = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": 1.0 / dt, "unit": "compressions/s", "cores": os.cpu_count(),
                                "kind": "port", "sample": "1 randcompress_adaptive of the same matrix"}
    print(json.dumps(line), flush=True)
    return 0


def run_matvec_workload(args):
    """HSS x dense product (``hss_matmul``, FP64) on the precision workload's tree
    (n = 65536, leafsize 128, k = 32): r = 1, where the product is bound by HBM
    bandwidth and GB300's FP64 rate, and r = --rhs.  The persistent product (one
    cooperative launch) is timed beside the level-by-level kernels.  L2 is flushed
    (512 MB write) before every timed call; CUDA events on the launching stream."""
    import numpy as np
    import torch
    import __graft_entry__ as g
    pkg = g.load_package()
    from hssmatrices_gb300 import synthetic as S
    n = args.n
    A = pkg.synthetic_hss(n, args.leafsize, args.rank, np.random.default_rng(args.seed))
    dev = A.device()
    lib = dev.lib
    entries = S.generator_entries(A)
    flush = torch.empty(512 * 1024 * 1024, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream()
    try:
        peak = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["hbm_gbs"])
        peak_src = "measured"
    except Exception:
        peak, peak_src = 6800.0, "fallback"
    out = {}
    clocks = Clocks(0)
    clocks.start()
    for r in sorted({1, args.rhs}):
        dB = torch.randn((r, n), dtype=torch.float64, device="cuda")
        dC = torch.empty_like(dB)
        alg = 8 * entries + 8 * r * (2 * n)     # generators + B read + C written
        res = {}
        for level in (0, 1):
            assert lib.hss_set_option(3, level) == 0
            try:
                for _ in range(max(3, args.warmup)):
                    dev.matmul_device(dB, n, r, dC, n, stream=stream)
                ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
                      for _ in range(args.steps)]
                torch.cuda.synchronize()
                for a, b in ev:
                    flush.zero_()
                    a.record(stream)
                    dev.matmul_device(dB, n, r, dC, n, stream=stream)
                    b.record(stream)
                torch.cuda.synchronize()
                t = sorted(x.elapsed_time(y) for x, y in ev)
                res["level" if level else "persistent"] = {
                    "us_median": 1000.0 * statistics.median(t), "us_min": 1000.0 * t[0],
                    "gbs": alg / (statistics.median(t) * 1e-3) / 1e9}
                res["C" if not level else "C_level"] = dC.cpu().numpy()
            finally:
                lib.hss_set_option(3, 0)
        diff = float(np.linalg.norm(res.pop("C") - res.pop("C_level")))
        out[r] = dict(res, algorithmic_bytes=alg, paths_rel_diff=diff / max(1e-300, float(torch.linalg.norm(dC))),
                      kernel="pmv_flat_kernel" if r <= 4 else "ozmv_kernel (tensor cores, one launch per level)")
    clk = clocks.stop()
    g1 = out[1]["persistent"]["gbs"]
    # full(hssA) on the device (src/hssmatrix.jl:270-305) for an n = 16384 tree
    # of the same construction: 2.1 GB written, 2 n^2 k FLOP of off-diagonal blocks
    nf = 16384
    hf = pkg.synthetic_hss(nf, args.leafsize, args.rank, np.random.default_rng(5)).device()
    Fo = torch.empty((nf, nf), dtype=torch.float64, device="cuda")
    for _ in range(2):
        pkg._lib.check(lib.hss_full(hf.handle, ctypes.c_void_p(Fo.data_ptr()), nf, None))
    torch.cuda.synchronize()
    tf = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        pkg._lib.check(lib.hss_full(hf.handle, ctypes.c_void_p(Fo.data_ptr()), nf, None))
        b.record()
        torch.cuda.synchronize()
        tf.append(a.elapsed_time(b))
    full_ms = statistics.median(tf)
    del Fo
    # HSS x HSS product (src/matmul.jl:65-117) of two n = 65536, k = 32 trees
    hb = pkg.synthetic_hss(n, args.leafsize, args.rank, np.random.default_rng(6)).device()
    hp = ctypes.c_void_p()
    th = []
    for it in range(4):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        pkg._lib.check(lib.hss_hssmul(dev.handle, hb.handle, ctypes.byref(hp), None))
        th.append(time.perf_counter() - t0)
        lib.hss_destroy(hp)
    hssmul_ms = 1000.0 * statistics.median(th[1:])
    # recompress! of that product (rank 64 -> its numerical rank at 1e-9)
    pkg._lib.check(lib.hss_hssmul(dev.handle, hb.handle, ctypes.byref(hp), None))
    hr = ctypes.c_void_p()
    tr = []
    for it in range(3):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        pkg._lib.check(lib.hss_recompress(hp, 1e-9, 1e-9, ctypes.byref(hr), None))
        tr.append(time.perf_counter() - t0)
        if it < 2:
            lib.hss_destroy(hr)
    recompress_ms = 1000.0 * statistics.median(tr[1:])
    info = (ctypes.c_int64 * 13)()
    pkg._lib.check(lib.hss_node_info(hr, 1, info))
    rec_rank = int(info[6])
    lib.hss_destroy(hr)
    lib.hss_destroy(hp)
    # hssA \ hssB (src/ulvdivide.jl:13) for two n = 16384 trees: expansion of B,
    # FP64 ULV solve of its 16384 columns, adaptive recompression to 1e-9
    hA = pkg.synthetic_hss(nf, args.leafsize, args.rank, np.random.default_rng(7))
    hB = pkg.synthetic_hss(nf, args.leafsize, args.rank, np.random.default_rng(8))
    hA.device(), hB.device()
    td = []
    for it in range(2):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        st = {}
        X = pkg.hss_ldiv(hA, hB, atol=1e-9, rtol=1e-9, stats=st)
        td.append(time.perf_counter() - t0)
    ldiv_rank = pkg.hssrank(X)
    del X
    leaf_flop = 2.0 * n * args.leafsize * args.leafsize * 2   # D_A D_B and the rank terms, leading order
    line = {
        "metric": "HSS matvec GB/s (FP64 hss_matmul, r=1)", "value": g1, "unit": "GB/s", "n_gpus": 1,
        "steps": args.steps, "warmup": max(3, args.warmup), "ms_per_step": out[1]["persistent"]["us_median"] / 1000.0,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": (f"matvec: synthetic HSS n={n}, perfect tree leafsize {args.leafsize}, k={args.rank}; "
                                f"C = A B with r = 1 and r = {args.rhs}; algorithmic bytes = 8 x generator entries "
                                f"({entries}) + 16 n r"), "l2": "flushed before every timed call (512 MB write)"},
        "roofline": {"kernel": "pmv_flat_kernel", "bound": "hbm", "achieved": g1, "peak": peak, "unit": "GB/s",
                     "frac": g1 / peak, "peak_source": peak_src,
                     "traffic": MATVEC_R1_TRAFFIC.get((n, args.leafsize, args.rank)),
                     "traffic_source": "ncu capture of one r = 1 launch at this size",
                     "note": "FP64 products of <= 4 columns run the flat persistent kernel, wide ones the tensor-core product"},
        "by_rhs": {str(r): v for r, v in out.items()}, "clocks": clk,
        "full_n16384": {"ms": full_ms, "written_gbs": nf * nf * 8 / (full_ms * 1e-3) / 1e9,
                        "fp64_tflops": 2.0 * nf * nf * args.rank / (full_ms * 1e-3) / 1e12},
        "hssmul_n65536": {"ms": hssmul_ms, "leaf_fp64_tflops": leaf_flop / (hssmul_ms * 1e-3) / 1e12,
                          "note": "host call to result handle (includes plan creation and the final synchronise)"},
        "recompress_product_n65536": {"ms": recompress_ms, "rank_in": 2 * args.rank, "rank_out_node1": rec_rank,
                                      "tol": 1e-9},
        "hss_ldiv_n16384": {"ms": 1000.0 * td[-1], "rank_out": ldiv_rank, "tol": 1e-9,
                            "note": "host call to result tree (FP64 ULV factor of A, the level-by-level "
                                    "recursion on the generators with recompression, copy to host)"},
    }
    print(json.dumps(line), flush=True)
    return 0


def run_steps(args):
    """Profiling aid: the precision workload's steps (FP32 factor + solve with
    refinement), --warmup + --steps of them, launched one by one (no graph
    replay, no autotuning, nothing timed), so that a profiler run on a few steps
    captures each kernel of a step as its own launch."""
    import numpy as np
    import torch
    import __graft_entry__ as g
    pkg = g.load_package()
    n, r = args.n, args.rhs
    A = pkg.synthetic_hss(n, args.leafsize, args.rank, np.random.default_rng(args.seed))
    dev = A.device()
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    dB = torch.from_numpy(np.ascontiguousarray(np.random.default_rng(1).standard_normal((n, r)).T)).cuda()
    dX = torch.zeros_like(dB)
    F = dev.ulvfactor("fp32", stream=stream)
    st = None
    for _ in range(args.warmup + args.steps):
        st = F.factsolve_device(dB, n, r, dX, n, tol=args.tol, maxit=20, stream=stream)
    torch.cuda.synchronize()
    print(json.dumps({"workload": "steps", "steps": args.warmup + args.steps, "iterations": st.iterations,
                      "residual": st.residual}), flush=True)
    return 0


def main():
    args = parse()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)
    if args.workload == "serve":
        return run_serve(args) if rank == 0 else 0
    if args.workload == "batch":
        return run_batch(args) if rank == 0 else 0
    if args.workload == "compress":
        return run_compress(args) if rank == 0 else 0
    if args.workload == "matvec":
        return run_matvec_workload(args) if rank == 0 else 0
    if args.workload == "steps":
        return run_steps(args) if rank == 0 else 0
    if world > 1:
        import torch
        import torch.distributed as td
        torch.cuda.set_device(local_rank)
        td.init_process_group("nccl")
    rc = run_ours(args, rank, world, local_rank)
    if world > 1:
        import torch.distributed as td
        td.destroy_process_group()
    return rc


if __name__ == "__main__":
    sys.exit(main())
