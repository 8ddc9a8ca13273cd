#!/usr/bin/env python
"""Benchmark of the variational ground-state sweep on B200.

Workload (config 2 of the measurement plan): spin-1/2 Heisenberg chain,
J = Jz = 1, hz = 0, open boundaries, L = 100, d = 2, Dw = 5, random uniform(-1,1)
seeded initial MPS; D schedule 16 -> 32 -> 64 -> 128 -> 256 expressed as the
reference's IterationSchedule lines {2,16,16},{2,32,16},{2,64,32},{2,128,64},
{2,256,128} (each line first re-runs the current D, MPSImp_Variational.C:33-40),
Krylov dimension 20, eigensolver tolerance 1e-10.

A "step" is the first sweep pair (Sweep(DLeft) + Sweep(DRight)) of the D = 256
schedule line: the state the D <= 128 lines converged is grown to D = 256 by
zero padding (MPSImp::IncreaseBondDimensions), uploaded, right-normalised with
its environments rebuilt (untimed), then swept once each way.  Every step
starts from the same snapshot, so the eigensolver does the same real work each
time.  `value` is device time per step (CUDA events on the library's launch
stream, max over ranks).  After the timed steps the D = 256 line is run to
convergence from the snapshot; the schedule's wall time and final energy are
reported too.  Inputs (site tensors plus environments, about
0.6 GB at D = 256) are larger than L2 between steps.

The headline path is the split-precision one (--precision mixed, the default).
Unless --no-fp64-compare is given, the plain FP64 GPU sweep runs the same
schedule from the same seed and is timed the same way; the line then carries
its time, the speed-up and the energy difference per site between the two.

Usage: python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                       [--precision fp64|mixed|mixed_hi] [--no-fp64-compare]
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "Sweep s and Heff TFLOP/s, L=100 D=256: mixed+learned vs FP64 GPU at ΔE/L≤1e-9"
L_CHAIN, S_SPIN, D_FINAL = 100, 0.5, 256
SCHEDULE = [(2, 16, 16), (2, 32, 16), (2, 64, 32), (2, 128, 64), (2, 256, 128)]
EPS_EIGEN = 1e-10
KRYLOV = 20
# DRAM bytes (read + write) of one Heff application, summed over its kernels, from
# the ncu capture of `bench.py --matvec-only --D 256` (profiles/heff_matvec_D256.md)
TRAFFIC = {("mixed", 256): 7.13e6, ("fp64", 256): 21.1e6}


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=3)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--precision", choices=["fp64", "mixed", "mixed_hi"], default="mixed")
    p.add_argument("--no-fp64-compare", action="store_true",
                   help="skip the FP64 GPU sweep on the same schedule (speed-up and energy check)")
    p.add_argument("--L", type=int, default=L_CHAIN)
    p.add_argument("--S", type=float, default=S_SPIN, help="spin (0.5: config 2; 1.0 with --L 128 --D 512: config 3)")
    p.add_argument("--D", type=int, default=D_FINAL)
    p.add_argument("--cpu-sites", type=int, default=4, help="bulk site updates in the CPU baseline sample")
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--mixed-tol", type=float, default=0.0,
                   help="split-precision Krylov residual target relative to |T| (0: the library default)")
    p.add_argument("--no-learned", action="store_true",
                   help="skip the Davidson arms (diagonal and learned correction) of the D step")
    p.add_argument("--ref-half-sweep", type=int, default=1,
                   help="reference arm: time one full half-sweep once to check the extrapolation (1) or not (0)")
    p.add_argument("--workload", choices=["sweep", "scan"], default="sweep",
                   help="scan: the XXZ parameter scan (independent chains, concurrent per-worker streams)")
    p.add_argument("--scan-n", type=int, default=64, help="scan instances (all ranks together)")
    p.add_argument("--scan-workers", type=int, default=8, help="concurrent contexts per GPU")
    p.add_argument("--scan-seq", type=int, default=8, help="instances timed sequentially for the comparison")
    p.add_argument("--matvec-only", action="store_true",
                   help="only time the bulk D x D Heff application through the operator handle (profiling)")
    p.add_argument("--profile-region", action="store_true",
                   help="bracket the timed steps with cudaProfilerStart/Stop (for ncu --profile-from-start off)")
    return p.parse_args()


def max_over_ranks(x, dist, device):
    """The slowest replica's time: every rank contributes its own device time."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def unit_of(args):
    return f"s per sweep pair (L={args.L}, D={args.D}{'' if args.S == 0.5 else f', S={args.S:g}'})"


def workload_of(args):
    d = int(round(2 * args.S + 1))
    return (f"Heisenberg S={args.S:g} L={args.L} open chain, d={d}, Dw=5: the first sweep pair of the D={args.D} line "
            f"(state converged by the D 16->{args.D // 2} schedule lines, 2 sweeps/line, then grown to D={args.D} "
            f"by zero padding), Krylov 20, eig tol 1e-10")


def grow_sites(sites, D):
    """MPSImp::IncreaseBondDimensions (MPSImp.C:123-147) on host arrays (d, D1, D2):
    zero-pad every site to the edge-aware ramp min(d^k, D) from both ends."""
    import numpy as np
    L, d = len(sites), sites[0].shape[0]
    dims = [None] * (L + 1)
    Dideal, ia = 1, 1
    while ia <= L // 2:
        dims[ia] = (min(Dideal, D), min(Dideal * d, D))
        Dideal = min(Dideal * d, D)
        ia += 1
    Dideal = 1
    for ib in range(L, ia - 1, -1):
        dims[ib] = (min(Dideal * d, D), min(Dideal, D))
        Dideal = min(Dideal * d, D)
    out = []
    for i, a in enumerate(sites, start=1):
        D1, D2 = dims[i]
        b = np.zeros((d, D1, D2))
        b[:, :a.shape[1], :a.shape[2]] = a
        out.append(b)
    return out


def schedule_for(D):
    lines = [ln for ln in SCHEDULE if ln[1] <= D]
    if not lines or lines[-1][1] != D:
        lines.append((2, D, max(1, D - (lines[-1][1] if lines else 16))))
    return lines


# ---------------------------------------------------------------------------
# clocks sampling (nvidia-smi during the timed region)
# ---------------------------------------------------------------------------
class ClockSampler:
    def __init__(self, index):
        self.index = index
        self.samples = []
        self._stop = threading.Event()
        self._proc = None

    def start(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self._proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                                           "--format=csv,noheader,nounits", "-lms", "200"],
                                          stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            threading.Thread(target=self._read, daemon=True).start()
        except Exception:
            self._proc = None

    def _read(self):
        for line in self._proc.stdout:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 9:
                self.samples.append(parts)

    def stop(self):
        if self._proc:
            self._proc.terminate()
            try:
                self._proc.wait(timeout=5)
            except Exception:
                self._proc.kill()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}
        sm = sorted(float(s[1]) for s in self.samples if s[1].replace(".", "").isdigit())
        mx = max((float(s[2]) for s in self.samples if s[2].replace(".", "").isdigit()), default=None)
        reasons = set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for s in self.samples:
            for nm, v in zip(names, s[5:9]):
                if v.strip().lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": sm[len(sm) // 2] if sm else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(self.samples)}


# ---------------------------------------------------------------------------
def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f), "measured"
    except Exception:
        return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0}, "fallback"


def fp64_peak_tflops(torch):
    """cuBLAS DGEMM 8192^3 (torch.matmul, float64) as the FP64 denominator, best of 5."""
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, n, dtype=torch.float64, device="cuda")
    for _ in range(2):
        torch.matmul(a, b)
    torch.cuda.synchronize()
    best = 1e9
    for _ in range(5):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        torch.matmul(a, b)
        e.record()
        e.synchronize()
        best = min(best, s.elapsed_time(e) / 1e3)
    del a, b
    return 2.0 * n ** 3 / best / 1e12


def qr_microbench(T, ctx, torch, m, n, reps=20):
    """Device time per thin QR (R and Q) of an m x n gauge matrix through tn_qr,
    CUDA events on the context's stream; returns (seconds, algorithmic flop)."""
    import ctypes as C
    lib = ctx._lib
    st = torch.cuda.current_stream()
    T._capi.check(lib.tn_ctx_set_stream(ctx.handle, C.c_void_p(st.cuda_stream)), "stream")
    k = min(m, n)
    A = torch.rand(m * n, dtype=torch.float64, device="cuda") * 2 - 1
    Q = torch.empty(m * k, dtype=torch.float64, device="cuda")
    R = torch.empty(k * n, dtype=torch.float64, device="cuda")

    def run():
        T._capi.check(lib.tn_qr(ctx.handle, m, n, A.data_ptr(), m, Q.data_ptr(), m, R.data_ptr(), k), "tn_qr")
    for _ in range(3):
        run()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        run()
    e1.record()
    torch.cuda.synchronize()
    T._capi.check(lib.tn_ctx_set_stream(ctx.handle, C.c_void_p(0)), "stream")
    # Householder R (2mn^2 - 2n^3/3) plus the thin Q formed from the reflectors (the same count)
    flop = 2.0 * (2.0 * m * k * k - 2.0 * k ** 3 / 3.0)
    return e0.elapsed_time(e1) / 1e3 / reps, flop


def heff_flops(d, Dw1, Dw2, D1, D2):
    return 2.0 * d * Dw1 * D1 * D1 * D2 + 2.0 * d * Dw2 * D1 * D2 * D2 + 2.0 * d * d * Dw1 * Dw2 * D1 * D2


def matvec_microbench(T, ctx, torch, D, precision, reps=50, S=0.5):
    """Average device time of one bulk Heff application at D x D (d=2, Dw=5) through
    the operator handle, on a torch stream that the library launches on, so that the
    torch events bracket exactly these launches."""
    import ctypes as C
    import numpy as np
    lib = ctx._lib
    H = T.Factory(ctx).Make1D_NN_HeisenbergHamiltonian(10, S, T.RegularLower, 1.0, 1.0, 0.0)
    W = np.ascontiguousarray(H.GetW(5).ravel())
    d, Dw = int(round(2 * S + 1)), 5
    g = torch.Generator(device="cuda").manual_seed(42)
    F = torch.rand(Dw * D * D, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    G = torch.rand(Dw * D * D, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    x = torch.rand(d * D * D, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    y = torch.empty_like(x)
    stream = torch.cuda.Stream()  # a real (non-default) stream shared by the library and the events
    torch.cuda.synchronize()
    lib.tn_ctx_set_stream(ctx.handle, stream.cuda_stream)
    try:
      with torch.cuda.stream(stream):
        prec = {"fp64": 0, "mixed": 1, "mixed_hi": 2}[precision]
        h = C.c_void_p()
        T._capi.check(lib.tn_heff_create(ctx.handle, prec, d, Dw, Dw, D, D, W.ctypes.data, F.data_ptr(),
                                         G.data_ptr(), C.byref(h)), "tn_heff_create")
        for _ in range(5):
            T._capi.check(lib.tn_heff_apply(h, x.data_ptr(), y.data_ptr()), "tn_heff_apply")
        torch.cuda.synchronize()
        # the applications recorded once in a CUDA graph and replayed, so that the
        # time is the device's and not the host's launch rate (eager loop if the
        # capture is refused)
        graph = None
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                for _ in range(reps):
                    T._capi.check(lib.tn_heff_apply(h, x.data_ptr(), y.data_ptr()), "tn_heff_apply")
            graph.replay()
            torch.cuda.synchronize()
        except Exception:
            graph = None
            torch.cuda.synchronize()
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record(stream)
        if graph is not None:
            graph.replay()
        else:
            for _ in range(reps):
                T._capi.check(lib.tn_heff_apply(h, x.data_ptr(), y.data_ptr()), "tn_heff_apply")
        e.record(stream)
        e.synchronize()
        t = s.elapsed_time(e) / 1e3 / reps
        del graph
        T._capi.check(lib.tn_heff_destroy(h), "tn_heff_destroy")
    finally:
        lib.tn_ctx_set_stream(ctx.handle, None)
    return t, heff_flops(d, Dw, Dw, D, D)


def lanczos_probe(T, ctx, D, peaks, d=2):
    """Achieved HBM bandwidth of the Lanczos Krylov kernels (CGS2 projections, update,
    next vector) at the bulk vector size N = 2 D^2, replayed from their CUDA graph on a
    diagonal operator (tn_lanczos_probe), against the measured copy bandwidth."""
    import ctypes as C
    N = d * D * D
    us, b = C.c_double(), C.c_double()
    T._capi.check(ctx._lib.tn_lanczos_probe(ctx.handle, N, KRYLOV, C.byref(us), C.byref(b)), "tn_lanczos_probe")
    gbs = b.value / (us.value * 1e-6) / 1e9
    return {"N": N, "krylov": KRYLOV, "us_per_step": round(us.value, 2), "bytes_per_step": round(b.value),
            "achieved_gbs": round(gbs, 1), "peak_gbs": peaks["hbm_gbs"], "frac": round(gbs / peaks["hbm_gbs"], 4),
            "note": "algorithmic bytes (j+4)N doubles per step j plus the diagonal operator's 2N; "
                    "device time from the graph replay (CUDA events)"}


def learned_arms(args, T, ctx, run_path, t_step, E_after, fp64_cmp):
    """Davidson on the same D step: diagonal correction, and the learned one (3-layer
    MLP, width 64, BF16 weights) trained on the GPU on exact corrections recorded from
    FP64 diagonal-Davidson sweeps of a small chain (L=16, D=32, 2 sweeps).  Diagonal
    Davidson is the judge: the energies after the step are compared."""
    f = T.Factory(ctx)
    Hs = f.Make1D_NN_HeisenbergHamiltonian(16, args.S, T.RegularLower, 1.0, 1.0, 0.0)
    t0 = time.perf_counter()
    ds = T.TrainingSet(2_000_000, ctx)
    psi = Hs.CreateMPS(32, 1e-12, 1e-12)
    psi.InitializeWith(T.Random, seed=21)
    psi.SetRecorder(ds)
    sched = T.IterationSchedule()
    eps = T.Epsilons(1e-12)
    eps.itsEigenSolverEpsilon = EPS_EIGEN
    sched.Insert(T.IterationScheduleLine(2, 32, 1, eps))
    psi.FindVariationalGroundState(Hs, sched, T.SolverOptions(eigensolver=T.DAVIDSON, krylov=16))
    psi.SetRecorder(None)
    F, Tt = ds.device_arrays()
    model = T.LearnedCorrection(seed=9, ctx=ctx)
    _, l0 = model.gradient(F, Tt)
    model.train(F, Tt, steps=1500, batch=4096, lr=2e-3, seed=3)
    _, l1 = model.gradient(F, Tt)
    train_s = time.perf_counter() - t0
    diag = run_path(args.precision, False, davidson=True, finish=False)
    lrn = run_path(args.precision, False, davidson=True, model=model, finish=False)
    ref = fp64_cmp["value"] if fp64_cmp else None
    return {"pairs": len(ds), "train_loss": [round(l0, 4), round(l1, 4)], "record_train_s": round(train_s, 2),
            "diagonal": {"value": round(diag["t_step"], 6), "matvecs_per_step": diag["matvecs"] / args.steps,
                         "dE_per_site_vs_lanczos": abs(diag["E_after"] - E_after) / args.L},
            "learned": {"value": round(lrn["t_step"], 6), "matvecs_per_step": lrn["matvecs"] / args.steps,
                        "dE_per_site_vs_diagonal": abs(lrn["E_after"] - diag["E_after"]) / args.L,
                        "learned_steps": lrn["last"].get("learned_steps"),
                        "fallbacks": lrn["last"].get("fallbacks")},
            "gain_matvecs_learned_vs_diagonal": round(diag["matvecs"] / max(lrn["matvecs"], 1), 3),
            "gain_time_learned_vs_diagonal": round(diag["t_step"] / lrn["t_step"], 3),
            "speedup_learned_vs_fp64_gpu": round(ref / lrn["t_step"], 3) if ref else None}


def run_ours(args, rank, world, local_rank):
    import ctypes as C

    import numpy as np
    import torch
    torch.cuda.set_device(local_rank)
    import tensornetworks_b200 as T

    dist = None
    if world > 1:
        import torch.distributed as dist
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))

    ctx = T.Context(local_rank)
    lib = ctx._lib
    f = T.Factory(ctx)
    H = f.Make1D_NN_HeisenbergHamiltonian(args.L, args.S, T.RegularLower, 1.0, 1.0, 0.0)
    lines = schedule_for(args.D)

    def run_path(precision, sample_clocks, fp64_tol_rel=0.0, davidson=False, model=None, finish=True):
        """Schedule up to the line before D, snapshot, then W warm-up and K timed steps;
        a step is the D line's first sweep pair from the grown snapshot."""
        prec = {"fp64": T.FP64, "mixed": T.MIXED, "mixed_hi": T.MIXED_HI}[precision]
        opts = T.SolverOptions(precision=prec, krylov=KRYLOV, max_restarts=10, fp64_tol_rel=fp64_tol_rel,
                               mixed_tol=args.mixed_tol)
        psi = H.CreateMPS(lines[0][1], 1e-12, 1e-12)
        psi.InitializeWith(T.Random, seed=1234)

        def make_sched(lns):
            sched = T.IterationSchedule()
            for (ms, Dm, dD) in lns:
                eps = T.Epsilons(1e-12)
                eps.itsEigenSolverEpsilon = EPS_EIGEN
                sched.Insert(T.IterationScheduleLine(ms, Dm, dD, eps))
            return sched

        t0 = time.perf_counter()
        if len(lines) > 1:
            psi.FindVariationalGroundState(H, make_sched(lines[:-1]), opts)
        pre_s = time.perf_counter() - t0
        grown = grow_sites([psi.GetSite(i) for i in range(1, args.L + 1)], args.D)
        if davidson:
            # the timed steps run Davidson (diagonal, or with the learned correction)
            opts = T.SolverOptions(precision=prec, eigensolver=T.DAVIDSON, krylov=16, max_restarts=10,
                                   use_learned=1 if model is not None else 0)
            psi.SetLearnedCorrection(model)

        def step():
            for i, a in enumerate(grown, start=1):
                psi.SetSite(i, a)
            psi.PrepareSweeps(H)
            return psi.Sweep(H, 1, EPS_EIGEN, opts)

        for _ in range(args.warmup):
            step()
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        clocks = ClockSampler(local_rank) if sample_clocks else None
        if clocks:
            clocks.start()
        launches0 = lib.tn_launch_count()
        step_ms, matvecs, flops = [], 0, 0.0
        if args.profile_region and sample_clocks:
            torch.cuda.profiler.start()
        for _ in range(args.steps):
            st = step()
            step_ms.append(st["sweep_ms"])
            matvecs += st["matvecs"]
            flops += st["heff_flop"]
        torch.cuda.synchronize()
        if args.profile_region and sample_clocks:
            torch.cuda.profiler.stop()
        launches = lib.tn_launch_count() - launches0
        if clocks:
            clocks.stop()
        t_step = max_over_ranks(sum(step_ms) / len(step_ms) / 1e3, dist, "cuda")
        # one more step, untimed, with CUDA events around every site's phases
        opts.phase_timing = 1
        ph = step()
        opts.phase_timing = 0
        phases = {"refine_ms": round(ph["refine_ms"], 3), "gauge_ms": round(ph["gauge_ms"], 3),
                  "env_ms": round(ph["env_ms"], 3), "sweep_ms": round(ph["sweep_ms"], 3)}
        if ph["sweep_ms"] > 0:
            phases["gauge_share"] = round(ph["gauge_ms"] / ph["sweep_ms"], 4)
            phases["refine_share"] = round(ph["refine_ms"] / ph["sweep_ms"], 4)
        E_step = psi.GetExpectation(H)
        last = dict(psi.last_stats)
        var = schedule_s = sched_stats = E_sched = None
        if finish:
            # finish the schedule (the D line to convergence) from the grown snapshot
            for i, a in enumerate(grown, start=1):
                psi.SetSite(i, a)
            t1 = time.perf_counter()
            var = psi.FindVariationalGroundState(H, make_sched([lines[-1]]), opts)
            schedule_s = pre_s + time.perf_counter() - t1
            sched_stats = dict(psi.last_stats)
            E_sched = psi.GetExpectation(H)
        return dict(psi=psi, opts=opts, var=var, schedule_s=schedule_s, sched_stats=sched_stats, E_sched=E_sched,
                    t_step=t_step, step_ms=step_ms, matvecs=matvecs, flops=flops, launches=launches,
                    clocks=clocks, E_after=E_step, grown=grown, step=step, last=last, phases=phases)

    main_run = run_path(args.precision, True)
    psi, opts, var = main_run["psi"], main_run["opts"], main_run["var"]
    t_step, step_ms, flops = main_run["t_step"], main_run["step_ms"], main_run["flops"]
    launches, clocks = main_run["launches"], main_run["clocks"]
    sched_stats, schedule_s = main_run["sched_stats"], main_run["schedule_s"]
    E_sched, E_after = main_run["E_sched"], main_run["E_after"]

    # --- end to end through the C ABI with host buffers, as a reference-side
    #     caller makes it: per step upload the grown snapshot from pinned host
    #     memory in the library's (oml) site layout, normalise + environments,
    #     one sweep pair, download every site into pinned host memory
    grown = main_run["grown"]
    lib, hmps = psi._lib, psi.handle
    up = []
    for a in grown:
        d_, D1_, D2_ = a.shape
        buf = torch.empty(a.size, dtype=torch.float64, pin_memory=True)
        buf.numpy()[:] = np.transpose(a, (0, 2, 1)).ravel()  # A(n, i1, i2) at n*D1*D2 + i2*D1 + i1
        up.append((D1_, D2_, buf))
    down = [torch.empty(a.size, dtype=torch.float64, pin_memory=True) for a in grown]
    h2d = sum(a.nbytes for a in grown)
    e2e_times, d2h = [], 0
    for _ in range(max(1, args.steps)):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for i, (D1_, D2_, buf) in enumerate(up, start=1):
            T._capi.check(lib.tn_mps_set_site(hmps, i, D1_, D2_, buf.data_ptr()), "tn_mps_set_site")
        psi.PrepareSweeps(H)
        psi.Sweep(H, 1, EPS_EIGEN, opts)
        d2h = 0
        for i in range(1, args.L + 1):
            D1c, D2c = C.c_int(), C.c_int()
            T._capi.check(lib.tn_mps_get_site_dims(hmps, i, C.byref(D1c), C.byref(D2c)), "dims")
            n_ = psi.d * D1c.value * D2c.value
            if down[i - 1].numel() < n_:
                down[i - 1] = torch.empty(n_, dtype=torch.float64, pin_memory=True)
            T._capi.check(lib.tn_mps_get_site(hmps, i, down[i - 1].data_ptr()), "tn_mps_get_site")
            d2h += 8 * n_
        e2e_times.append(time.perf_counter() - t0)
    e2e = sum(e2e_times) / len(e2e_times)

    # --- the plain FP64 GPU sweep on the same schedule and seed
    fp64_cmp = None
    if args.precision != "fp64" and not args.no_fp64_compare:
        ref64 = run_path("fp64", False)
        fp64_cmp = {"value": round(ref64["t_step"], 6), "unit": unit_of(args),
                    "speedup": round(ref64["t_step"] / t_step, 3),
                    "schedule_s": round(ref64["schedule_s"], 3),
                    "energy_per_bond": ref64["E_after"] / (args.L - 1),
                    "dE_per_site_schedule": abs(E_sched - ref64["E_sched"]) / args.L,
                    "dE_per_site_after_steps": abs(E_after - ref64["E_after"]) / args.L,
                    "matvecs_per_step": ref64["matvecs"] / args.steps,
                    "phases_device_ms": ref64["phases"]}
        del ref64
        # the FP64 sweep stopped by the split-precision path's rule: residual relative
        # to |T| (2e-6, 1e-9 for mixed_hi) with the stall test, so that the speed-up
        # from precision is separated from the speed-up from the stop rule
        tol_rel = args.mixed_tol if args.mixed_tol > 0 else (1e-9 if args.precision == "mixed_hi" else 2e-6)
        same = run_path("fp64", False, fp64_tol_rel=tol_rel, finish=False)
        fp64_cmp["same_stop_rule"] = {
            "value": round(same["t_step"], 6), "unit": unit_of(args), "fp64_tol_rel": tol_rel,
            "speedup_of_split_precision": round(same["t_step"] / t_step, 3),
            "speedup_over_fp64_tol_1e-10": round(fp64_cmp["value"] / same["t_step"], 3),
            "dE_per_site_vs_split_precision": abs(E_after - same["E_after"]) / args.L,
            "matvecs_per_step": same["matvecs"] / args.steps,
            "phases_device_ms": same["phases"]}
        del same

    learned = None
    if not args.no_learned:
        learned = learned_arms(args, T, ctx, run_path, t_step, E_after, fp64_cmp)

    # --- roofline of the dominant kernel (the bulk Heff contraction chain)
    t_mv, F_mv = matvec_microbench(T, ctx, torch, args.D, args.precision, S=args.S)
    peaks, peak_kind = measured_peaks()
    if args.precision == "fp64":
        peak = fp64_peak_tflops(torch)
        peak_src = "cuBLAS DGEMM 8192^3 measured in this run"
    else:
        nprod = 3 if args.precision == "mixed" else 6
        peak = peaks["bf16_tflops"] / nprod
        peak_src = f"{peak_kind} bf16 burst / {nprod} (BF16 split products per FP32-accurate flop)"
    achieved = F_mv / t_mv / 1e12
    # DRAM bytes per application from the ncu capture of the same command
    # (profiles/heff_matvec_D256.md); measured at D = 256 only
    traffic = TRAFFIC.get((args.precision, args.D))
    roofline = {"bound": "tensor", "achieved": round(achieved, 3), "peak": round(peak, 2), "unit": "TFLOP/s",
                "frac": round(achieved / peak, 4), "traffic": traffic,
                "kernel": "heff_matvec (x split + two segmented tcgen05 GEMMs)" if args.precision != "fp64"
                else "heff_matvec (FP64 DMMA chain)",
                "per_launch_us": round(t_mv * 1e6, 2), "flop_per_launch": F_mv, "peak_source": peak_src}

    lanczos = lanczos_probe(T, ctx, args.D, peaks, d=int(round(2 * args.S + 1)))

    # --- the kernel with the largest share of the step: the gauge QR of a bulk
    #     site (d D x D), latency-bound (a chain of dependent column steps)
    d_ = int(round(2 * args.S + 1))
    t_qr, F_qr = qr_microbench(T, ctx, torch, d_ * args.D, args.D)
    p64 = fp64_peak_tflops(torch)
    ph = main_run["phases"] or {}
    roofline_qr = {"bound": "fp64 (latency)", "achieved": round(F_qr / t_qr / 1e12, 4), "peak": round(p64, 2),
                   "unit": "TFLOP/s", "frac": round(F_qr / t_qr / 1e12 / p64, 5), "traffic": None,
                   "kernel": f"gauge QR of a {d_ * args.D} x {args.D} site matrix (tn_qr: cluster Householder "
                             "kernel; the sweep's own gauge moves keep the persistent kernel's order)" if d_ * args.D <= 512 else
                             f"gauge QR of a {d_ * args.D} x {args.D} site matrix (tn_qr)",
                   "per_launch_us": round(t_qr * 1e6, 1), "flop_per_launch": F_qr,
                   "share_of_step": ph.get("gauge_share"),
                   "peak_source": "cuBLAS DGEMM 8192^3 measured in this run"}

    out = None
    if rank == 0:
        cpu = None
        if not args.no_cpu:
            cpu = cpu_baseline_same_state(args, grown, step_ms, psi)
        clk = clocks.summary()
        out = {
            "metric": METRIC,
            "value": round(t_step, 6),
            "unit": unit_of(args),
            "n_gpus": world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": round(t_step * 1e3, 3),
            "higher_is_better": False,
            "scaling": "weak",
            "vs_baseline": None,
            "dtype": {"fp64": "f64", "mixed": "bf16x3 (f32 acc) contractions, f64 Lanczos/QR/SVD/energies",
                      "mixed_hi": "bf16x6 (f32 acc) contractions, f64 Lanczos/QR/SVD/energies"}[args.precision],
            "data": "synthetic (seeded uniform(-1,1) initial MPS)",
            "config": {"workload": workload_of(args),
                       "precision": args.precision, "parallelism": f"replicas x{world}",
                       "l2": "inputs > L2 (site tensors + environments ~ 0.6 GB at D=256)"},
            "heff_tflops_sweep": round(flops / (sum(step_ms) / 1e3) / 1e12, 4),
            "matvecs_per_step": main_run["matvecs"] / args.steps,
            "phases_device_ms": main_run["phases"],
            "fp64_gpu": fp64_cmp,
            "schedule_s": round(schedule_s, 3),
            "schedule_sweep_ms": round(sched_stats["sweep_ms"], 1),
            "energy_per_bond": E_after / (args.L - 1),
            "energy_schedule_per_bond": E_sched / (args.L - 1),
            "variance": var,
            "e2e": {"value": round(e2e, 6), "unit": unit_of(args), "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h},
            "gpu_launches": int(launches),
            "roofline": roofline,
            "roofline_gauge_qr": roofline_qr,
            "lanczos_hbm": lanczos,
            "davidson_learned": learned,
            "cpu_baseline": cpu,
            "clocks": clk,
        }
        print(json.dumps(out), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    return out


def run_scan_bench(args, rank, world, local_rank):
    """XXZ parameter scan: the instances are partitioned over ranks (no data-path
    collective); each rank solves its share with concurrent per-worker contexts.
    The value is instances per second of the whole job (max wall time over
    ranks); the sequential rate is measured on the first --scan-seq instances
    of rank 0 with a single context."""
    import torch
    import tensornetworks_b200 as T
    from tensornetworks_b200 import scan
    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))
    allinst = scan.make_xxz_scan(args.scan_n, seed=777)
    mine = allinst[rank::world]
    opts = T.SolverOptions(precision={"fp64": T.FP64, "mixed": T.MIXED, "mixed_hi": T.MIXED_HI}[args.precision])
    # warm-up: one small instance per worker context shape
    scan.run_scan(mine[:1], workers=1, device=local_rank, options=opts)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    res, wall = scan.run_scan(mine, workers=args.scan_workers, device=local_rank, options=opts)
    torch.cuda.synchronize()
    wall = max_over_ranks(wall, dist, "cuda")
    seq = sub_par = None
    if rank == 0 and args.scan_seq > 0:
        sub = mine[:args.scan_seq]
        _, t_seq = scan.run_scan(sub, workers=1, device=local_rank, options=opts)
        _, t_sub = scan.run_scan(sub, workers=args.scan_workers, device=local_rank, options=opts)
        seq, sub_par = len(sub) / t_seq, len(sub) / t_sub
    if rank == 0:
        value = len(allinst) / wall
        out = {"metric": "XXZ parameter scan throughput", "value": round(value, 4), "unit": "instances/s",
               "n_gpus": world, "steps": 1, "warmup": 1, "ms_per_step": round(wall * 1e3, 1),
               "higher_is_better": True, "scaling": "strong" if world > 1 else "weak", "vs_baseline": None,
               "dtype": args.precision, "data": "synthetic (seeded XXZ instances, seed 777)",
               "config": {"workload": f"{len(allinst)} XXZ chains, Jz~U[-0.5,1.5], hz~U[0,0.5], L~U{{32..96}}, "
                                      f"D~U{{32,64,128}}, schedule D 16->D doubling (2 sweeps/line)",
                          "parallelism": f"{world} GPU(s) x {args.scan_workers} concurrent contexts",
                          "precision": args.precision},
               "sequential_instances_per_s": round(seq, 4) if seq else None,
               "subset_concurrent_instances_per_s": round(sub_par, 4) if sub_par else None,
               "speedup_vs_sequential_same_subset": round(sub_par / seq, 3) if seq else None,
               "energies_per_site": [round(r.energy_per_site, 10) for r in res][:8]}
        print(json.dumps(out), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def cpu_baseline_same_state(args, sites, step_ms, psi):
    """The oracle (FP64 C++ restatement, OpenMP on all host cores) timed on the same
    MPS for a bounded sample of bulk site updates, scaled to a sweep pair by the
    algorithmic Heff cost of every site."""
    from oracle import oracle as O
    ncores = os.cpu_count() or 1
    first = args.L // 2 - args.cpu_sites // 2
    sec, nmv = O.sweep_sample(args.L, args.S, sites, first, args.cpu_sites, krylov=KRYLOV, max_restarts=10,
                              tol=EPS_EIGEN, nthreads=ncores)
    per_site = sec / args.cpu_sites
    d, Dw = int(round(2 * args.S + 1)), 5
    bulk = heff_flops(d, Dw, Dw, args.D, args.D)
    w = 0.0
    for a in sites:
        D1, D2 = a.shape[1], a.shape[2]
        w += heff_flops(d, Dw, Dw, D1, D2) / bulk
    est = per_site * 2.0 * w
    return {"value": round(est, 3), "unit": unit_of(args), "cores": ncores, "kind": "port",
            "sample": f"{args.cpu_sites} bulk D={args.D} site updates (Lanczos Krylov 20 tol 1e-10 + QR gauge + "
                      f"environment) of the same grown snapshot the GPU step starts from, in {sec:.2f}s ({nmv} "
                      f"matvecs); scaled by the Heff cost of all 2L site updates of a sweep pair"}


def reference_snapshot(args):
    """The input of the timed step: the state the D <= D/2 schedule lines converge to
    from seed 1234, grown to D by zero padding -- the same snapshot the GPU arm
    starts from.  It is prepared (untimed) by the library's FP64 path when a GPU is
    present; otherwise a random right-canonical MPS of the same shapes stands in."""
    import numpy as np
    try:
        import torch
        gpu = torch.cuda.is_available()
    except Exception:
        gpu = False
    if gpu:
        import tensornetworks_b200 as T
        ctx = T.Context(0)
        H = T.Factory(ctx).Make1D_NN_HeisenbergHamiltonian(args.L, args.S, T.RegularLower, 1.0, 1.0, 0.0)
        lines = schedule_for(args.D)
        psi = H.CreateMPS(lines[0][1], 1e-12, 1e-12)
        psi.InitializeWith(T.Random, seed=1234)
        sched = T.IterationSchedule()
        for (ms, Dm, dD) in lines[:-1]:
            eps = T.Epsilons(1e-12)
            eps.itsEigenSolverEpsilon = EPS_EIGEN
            sched.Insert(T.IterationScheduleLine(ms, Dm, dD, eps))
        if len(lines) > 1:
            psi.FindVariationalGroundState(H, sched, T.SolverOptions(precision=T.FP64, krylov=KRYLOV))
        sites = grow_sites([psi.GetSite(i) for i in range(1, args.L + 1)], args.D)
        del psi, H
        ctx.close()
        return sites, True
    L, D, d = args.L, args.D, int(round(2 * args.S + 1))
    rng = np.random.default_rng(1234)
    sites = []
    for i in range(L):
        l = 1 if i == 0 else min(D, d ** i, d ** (L - i))
        r = 1 if i == L - 1 else min(D, d ** (i + 1), d ** (L - i - 1))
        sites.append(rng.uniform(-1, 1, size=(d, l, r)))
    return sites, False


def run_reference(args, rank, world):
    """The reference's CPU algorithm for the path: the oracle restatement (the reference
    itself cannot be built: its oml/LAPACK/ARPACK/PRIMME dependencies are absent), on
    all host cores, on the same snapshot as the GPU arm.  A step is a bounded sample of
    --cpu-sites bulk site updates, extrapolated to a sweep pair by the Heff cost of
    every site; once per run a full half-sweep (all L-1 updates) is timed as well, as
    the check of that extrapolation."""
    if rank != 0:
        return None
    from oracle import oracle as O
    O.build()
    ncores = os.cpu_count() or 1
    L, D, d = args.L, args.D, int(round(2 * args.S + 1))
    sites, same = reference_snapshot(args)
    first = L // 2 - args.cpu_sites // 2
    bulk = heff_flops(d, 5, 5, D, D)
    w = sum(heff_flops(d, 5, 5, a.shape[1], a.shape[2]) / bulk for a in sites)
    if args.warmup > 0:  # one untimed site update (page-in, thread start)
        O.sweep_sample(L, args.S, sites, first, 1, krylov=KRYLOV, max_restarts=10, tol=EPS_EIGEN, nthreads=ncores)
    times = []
    for _ in range(max(1, args.steps)):
        sec, nmv = O.sweep_sample(L, args.S, sites, first, args.cpu_sites, krylov=KRYLOV, max_restarts=10,
                                  tol=EPS_EIGEN, nthreads=ncores)
        times.append(sec)
    per_site = sum(times) / len(times) / args.cpu_sites
    value = per_site * 2.0 * w
    check = None
    if args.ref_half_sweep:
        sec, nmv = O.sweep_sample(L, args.S, sites, 1, L - 1, krylov=KRYLOV, max_restarts=10, tol=EPS_EIGEN,
                                  nthreads=ncores)
        w_half = sum(heff_flops(d, 5, 5, a.shape[1], a.shape[2]) / bulk for a in sites[:L - 1])
        check = {"half_sweep_measured_s": round(sec, 3), "half_sweep_extrapolated_s": round(per_site * w_half, 3),
                 "ratio_measured_over_extrapolated": round(sec / (per_site * w_half), 3), "matvecs": nmv,
                 "sweep_pair_from_measured_half_s": round(2.0 * sec, 3)}
    sample = (f"{args.cpu_sites} bulk D={D} site updates (Lanczos Krylov 20 tol 1e-10 + QR gauge + environment) "
              f"of the {'same grown snapshot the GPU arm starts from (prepared untimed by the library FP64 path)' if same else 'random right-canonical MPS of the same shapes (no GPU to prepare the snapshot)'} "
              f"per step, extrapolated to the 2L site updates of a sweep pair by their Heff cost; oracle C++ "
              f"restatement (reference not buildable here)")
    out = {"metric": METRIC, "value": round(value, 3), "unit": unit_of(args),
           "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(value * 1e3, 1),
           "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
           "data": "synthetic", "impl": "reference", "same_config": same,
           "extrapolated_from_site_updates": args.cpu_sites,
           "config": {"workload": workload_of(args), "precision": "fp64 (CPU oracle restatement)"},
           "half_sweep_check": check,
           "cpu_baseline": {"value": round(value, 3), "unit": unit_of(args), "cores": ncores, "kind": "port",
                            "sample": sample},
           "e2e": {"value": round(value, 3), "unit": unit_of(args), "h2d_bytes_per_step": 0,
                   "d2h_bytes_per_step": 0}}
    print(json.dumps(out), flush=True)
    return out


def main():
    args = parse()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", str(args.gpus if args.gpus else 1)))
    if "WORLD_SIZE" not in os.environ:
        world = 1
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
    elif args.workload == "scan":
        run_scan_bench(args, rank, world, local_rank)
    elif args.matvec_only:
        import torch
        import tensornetworks_b200 as T
        torch.cuda.set_device(local_rank)
        t, flop = matvec_microbench(T, T.Context(local_rank), torch, args.D, args.precision, reps=max(1, args.steps),
                                    S=args.S)
        print(json.dumps({"matvec_us": round(t * 1e6, 2), "flop": flop, "tflops": round(flop / t / 1e12, 3),
                          "D": args.D, "precision": args.precision}), flush=True)
    else:
        run_ours(args, rank, world, local_rank)


if __name__ == "__main__":
    main()
