#!/usr/bin/env python
"""Wind solves/s of the B200 iterative wind solver on a seeded synthetic
terrain case (the 512 x 512 x 48 plain-BiCGStab workload).

One step = one steady-state wind solve of HICAR's update_winds path
(wind.F90:805-807): calc_divergence of fresh winds, then calc_iter_winds
(RHS, BiCGStab to 1e-6 relative residual with the probed operator, lambda ->
u/v/w correction).  The operator is calibrated once before timing, as HICAR
does on its first wind update; every step starts from lambda = 0 and the same
input winds.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

N > 1 runs one independent subdomain per rank (weak scaling, no collective on
the data path; torch.distributed only for the barrier and the max-over-ranks
timing).  --impl reference times the CPU restatement of the reference solver
(the reference itself cannot be compiled here) on a bounded sample of the same
workload on the host cores.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "wind solves/s to 1e-6 rel. residual, learned+mixed vs plain BiCGStab, 1 B200"
UNIT = "solves/s"
WORKLOADS = {
    "plain512": dict(nx=512, ny=512, nz=48, dx=250.0, n_hills=20, alpha="const", adv_den=True),
    "cpu64": dict(nx=64, ny=64, nz=20, dx=250.0, n_hills=20, alpha="const", adv_den=True),
    # a smaller case whose inputs still exceed L2, for ncu captures
    "mid256": dict(nx=256, ny=256, nz=48, dx=250.0, n_hills=20, alpha="const", adv_den=True),
    # 67 M cells, 60 hills, alpha a smooth seeded field in [0.3, 1.0]
    "mixed1024": dict(nx=1024, ny=1024, nz=64, dx=250.0, n_hills=60, alpha="smooth", adv_den=True),
    # the learned preconditioner's training grid (its parameters come from seeds 1000..1015;
    # the bench case, seed 1, is unseen) and its larger evaluation domain
    "learn128": dict(nx=128, ny=128, nz=32, dx=250.0, n_hills=20, alpha="const", adv_den=True),
    "eval768": dict(nx=768, ny=1536, nz=48, dx=250.0, n_hills=20, alpha="const", adv_den=True),
    # 96 independent subdomains, nx, ny in 96..512 step 32, nz in 20..48 step 4 (seeded), solved
    # together by the batched graph solver (one step = all 96 solves)
    "batch12": dict(batch=12, nxy=(96, 256, 32), nz=(20, 32, 4), dx=250.0, n_hills=20, alpha="const", adv_den=True),
    "batch96": dict(batch=96, nxy=(96, 512, 32), nz=(20, 48, 4), dx=250.0, n_hills=20, alpha="const", adv_den=True),
}
# BiCGStab iterations the CPU restatement (2-sweep Jacobi-Richardson, FP64
# Krylov, probed operator, 1e-6 recurrence norm) needs on each workload's
# seed-1 case, measured by running it to convergence on the host (plain512:
# 912 iterations, 136 s on 8 cores); the CPU sample extrapolates one solve
# from these.
# mixed1024: 1245, the count of the same method (plain BiCGStab, FP64 Krylov) on the GPU.
REF_ITERS_SOURCE = {"plain512": "the CPU oracle run to convergence on the host (912 iterations)",
                    "cpu64": "the CPU oracle run to convergence on the host (78 iterations)",
                    "mixed1024": "the same method (reference BiCGStab, FP64 Krylov, 2-sweep Jacobi-Richardson) "
                                 "run to convergence on the GPU on this case (1245 iterations; about 13 min on "
                                 "the host cores)"}
REF_ITERS = {"plain512": 912, "cpu64": 78, "mid256": None, "mixed1024": 1245, "learn128": None, "eval768": None, "batch12": None, "batch96": None}
# DRAM bytes per interior cell of one launch of the dominant kernel, from one
# ncu capture on a smaller case (the kernel reads and writes each cell's data
# once, so its traffic scales with the cells of the workload), keyed by the
# kernel and whether the Krylov vectors it reads and writes are FP64:
# mg_post_l0 with FP32 vectors, 255.41 MB per launch at 256x256x48 (3145728
# cells).  None for the FP64-vector form and the register-fed smoother
# (HICARW_MG_TMA=0), which were not captured in their current form.
TRAFFIC_PER_CELL = {} if os.environ.get("HICARW_MG_TMA", "2")[:1] in ("0", "1") else {
    ("mg_post_l0", False): (245.309696e6 + 10.103296e6) / (256 * 256 * 48)}
TOL = 1.0e-6
MG_COARSE_SCALE = None  # --mg-coarse-scale
MG_OMEGA = None  # --mg-omega
MG_SKIP_FINE_PRE = False  # --mg-skip-fine-presmooth
MG_W_LEVELS = ()  # --mg-w-levels
FGMRES_RESTART = None  # --fgmres-restart


def bf16_sustained():
    """Measured sustained dense BF16 TFLOP/s of this pool's B200s (None if not recorded)."""
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            return float(json.load(f).get("bf16_tflops_sustained") or 0.0) or None
    return None


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            j = json.load(f)
        return float(j["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


# Cycle shapes among which the mg preset picks on the problem at hand (in the
# untimed warm-up): the V-cycle with pre- and post-smoothing on every level
# (omega 0.8), V(0,1) on the finest level with omega 1, and the same with two
# coarse-grid corrections (a W-cycle) on levels 2-3, 2-4, 3-4, 3-5 or 4-5.
MG_CYCLES = {
    "V11": dict(),
    "V01": dict(mg_skip_fine_presmooth=True, mg_omega=1.0),
    "V01-W23": dict(mg_skip_fine_presmooth=True, mg_omega=1.0, mg_w_levels=(2, 3)),
    "V01-W24": dict(mg_skip_fine_presmooth=True, mg_omega=1.0, mg_w_levels=(2, 3, 4)),
    "V01-W34": dict(mg_skip_fine_presmooth=True, mg_omega=1.0, mg_w_levels=(3, 4)),
    "V01-W35": dict(mg_skip_fine_presmooth=True, mg_omega=1.0, mg_w_levels=(3, 4, 5)),
    "V01-W45": dict(mg_skip_fine_presmooth=True, mg_omega=1.0, mg_w_levels=(4, 5)),
}
MG_CYCLE = "auto"  # --mg-cycle
KRYLOV_F32_X64 = 2  # hicarw.h: FP32 Krylov vectors, FP64 reductions and lambda


def krylov_desc(opt) -> str:
    """Krylov arithmetic of a solve's options, for the bench line."""
    return {0: "f64", 1: "f32 vectors, f64 reductions",
            KRYLOV_F32_X64: "f32 vectors, f64 reductions and lambda"}.get(int(opt.krylov_precision), "f64")


def _timed_solve(wi, step, kw):
    """Set the options, run one solve (graph capture), time a second one with
    CUDA events; (ms, stats) of the timed one."""
    import torch
    wi.set_options(wi.WindOptions(**kw))
    step()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    st = step()
    e1.record()
    torch.cuda.synchronize()
    return round(e0.elapsed_time(e1), 3), st


def pick_cycle(wi, step, base: dict):
    """Two solves of the workload with each cycle of MG_CYCLES (the second one
    timed), then the fastest of them once more with FP32 Krylov vectors and
    FP64 lambda, and the faster of those with the finest level's smoother
    coefficients in BF16 (cycles without fine pre-smoothing).  Returns
    the options of the fastest candidate that converged with the multigrid
    preconditioner (no fallback) and, for the last two, whose FP64 true
    residual meets the tolerance; its name; and the table of times (ms; None
    for a candidate that was not accepted)."""
    table = {}
    for name, kw in MG_CYCLES.items():
        ms, st = _timed_solve(wi, step, {**base, **kw})
        table[name] = ms if st["status"] == 0 and st["precond"] == 1 else None
    good = {k: v for k, v in table.items() if v is not None}
    best = min(good, key=good.get) if good else "V11"
    kw = {**base, **MG_CYCLES[best]}
    if good:
        best_ms = table[best]
        # the same cycle with FP32 Krylov vectors and FP64 lambda
        trials = [("f32-vectors", {"krylov_precision": KRYLOV_F32_X64})]
        if kw.get("mg_skip_fine_presmooth"):  # BF16 coefficients of the finest level's post-smoother
            trials.append(("bf16-smoother", {"mg_precision": 1}))
        for tag, extra in trials:
            trial = {**kw, **extra}
            ms, st = _timed_solve(wi, step, trial)
            ok = st["status"] == 0 and st["precond"] == 1 and 0.0 <= st["true_res"] <= 1.01 * st["target"]
            table[best + "/" + tag] = ms if ok else None
            if ok and ms < best_ms:
                best, kw, best_ms = best + "/" + tag, trial, ms
    opt = wi.WindOptions(**kw)
    wi.set_options(opt)
    return opt, best, table


def solver_kwargs(name: str) -> dict:
    """WindOptions keyword arguments of a solver preset (with the command-line overrides)."""
    from hicar_b200 import _capi
    presets = {
        # the reference's method and kernel schedule, FP64 Krylov vectors
        "plain": dict(solver=_capi.SOLVER_REFERENCE, krylov_precision=_capi.KRYLOV_F64),
        # same BiCGStab recurrences, FP32 multigrid V-cycle preconditioner, true-residual stop,
        # the reference solve as the fallback on a 1%-per-50-iterations stall
        "mg": dict(solver=_capi.SOLVER_REFERENCE, krylov_precision=_capi.KRYLOV_F64,
                   precond=_capi.PRECOND_MG, stall_iters=50),
        # flexible GMRES(30) outer loop around the same V-cycle, FP64 Arnoldi basis
        "fgmres": dict(solver=_capi.SOLVER_FGMRES, precond=_capi.PRECOND_MG, fgmres_restart=30),
        # flexible GMRES(30) with the reference Jacobi-Richardson preconditioner (A/B baseline)
        "fgmres_jacobi": dict(solver=_capi.SOLVER_FGMRES, precond=_capi.PRECOND_JACOBI, fgmres_restart=30),
        # flexible GMRES(30) with the trained U-Net preconditioner (BF16 tensor-core
        # convolutions), the reference solve as the fallback on a stall
        "learned": dict(solver=_capi.SOLVER_FGMRES, precond=_capi.PRECOND_LEARNED, fgmres_restart=30,
                        stall_iters=100),
    }
    kw = dict(presets[name])
    if MG_COARSE_SCALE is not None and "precond" in kw:
        kw["mg_coarse_scale"] = MG_COARSE_SCALE
    if MG_OMEGA is not None and "precond" in kw:
        kw["mg_omega"] = MG_OMEGA
    if MG_SKIP_FINE_PRE and "precond" in kw:
        kw["mg_skip_fine_presmooth"] = True
    if MG_W_LEVELS and "precond" in kw:
        kw["mg_w_levels"] = tuple(MG_W_LEVELS)
    if FGMRES_RESTART is not None and "fgmres_restart" in kw:
        kw["fgmres_restart"] = FGMRES_RESTART
    return dict(tol_rel=TOL, wind_solver_iterations=3000, **kw)


def solver_options(name: str):
    from hicar_b200 import wind_iterative as wi
    return wi.WindOptions(**solver_kwargs(name))


# parts of the line that are tables or say at length what other keys say: in the file of the whole line only
LONG_PARTS = (("roofline", "kernels"), ("config", "accuracy"), ("config", "learned_fgmres"),
              ("config", "mg_cycle", "warmup_solve_ms"), ("config", "kernel_autotune"), ("batch96", "config"))


def print_line(line: dict) -> None:
    """The bench line on stdout, short enough to be read from the end of a log: without the long parts and
    with seven digits.  build/bench_line.json (config.whole_line) holds it whole."""
    path = os.path.join("build", "bench_line.json")
    try:
        os.makedirs(os.path.join(ROOT, "build"), exist_ok=True)
        with open(os.path.join(ROOT, path), "w") as f:
            json.dump(line, f, indent=1)
    except OSError:
        path = None

    def short(x, at=()):
        if isinstance(x, dict):
            return {k: short(v, at + (k,)) for k, v in x.items() if at + (k,) not in LONG_PARTS}
        if isinstance(x, (list, tuple)):
            return [short(v, at) for v in x]
        return float("%.7g" % x) if isinstance(x, float) else x

    out = short(line)
    out["config"]["whole_line"] = path
    print(json.dumps(out), flush=True)


class ClockSampler:
    """nvidia-smi samples during the timed region (never changes a setting)."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        with open(self.path) as f:
            for line in f:
                p = [x.strip() for x in line.split(",")]
                if len(p) < 9:
                    continue
                try:
                    sm.append(float(p[1]))
                    smax.append(float(p[2]))
                except ValueError:
                    continue
                for n, v in zip(names, p[5:9]):
                    if v.lower() == "active":
                        reasons.add(n)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "samples": len(sm), "reasons": sorted(reasons)}


def dist_setup():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def reduce_max(value: float, dist, device) -> float:
    """The maximum of `value` over all ranks (the job's time is the slowest rank's)."""
    if not dist:
        return value
    import torch
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def subdomain_seed(rank: int) -> int:
    """Each rank solves its own independent subdomain(s): seeds 1, 2, ... by rank."""
    return 1 + rank


def build_inputs(wl: dict, seed: int):
    from hicar_b200 import cases
    return cases.build_case(wl["nx"], wl["ny"], wl["nz"], wl["dx"], wl["n_hills"], seed=seed,
                            adv_den=wl["adv_den"], alpha=wl["alpha"])


# --------------------------------------------------------------------------------------
# CPU restatement, bounded sample (reference arm, and cpu_baseline of our arm)
# --------------------------------------------------------------------------------------
class CpuSample:
    """The CPU oracle (reference precision, OpenMP over j-planes) on one
    steady-state solve of `case`, sampled: divergence, RHS/diagonal,
    `sample_iters` BiCGStab iterations and the lambda -> wind correction are
    timed in full; the solve time is extrapolated to `ref_iters` iterations.
    The probed operator is calibrated on the CPU (or handed in) before timing;
    `solver` reuses an oracle solver that already holds it."""

    def __init__(self, case, coefs=None, threads=None, solver=None):
        import numpy as np
        from oracle import oracle as O
        O.build()
        if threads:
            O.set_threads(threads)
        self.np = np
        self.case = case
        self.cores = O.lib("ref").orc_get_threads()
        t = time.perf_counter()
        if solver is not None:
            self.s = solver
        else:
            self.s = O.OracleSolver(case.domain, "ref")
            self.s.set_alpha(case.alpha)
            if coefs is None:
                u, v, w = (np.ascontiguousarray(a).copy() for a in (case.u, case.v, case.w))
                self.s.build_analytic(case.alpha)
                self.s.calibrate(case.adv_den, u, v, w)
            else:
                self.s.set_coefs(coefs, probed=True)
        self.setup_s = time.perf_counter() - t

    def run(self, ref_iters, sample_iters):
        np, s, case = self.np, self.s, self.case
        u, v, w = (np.ascontiguousarray(a).copy() for a in (case.u, case.v, case.w))
        t0 = time.perf_counter()
        div = s.divergence(u, v, w, adv_den=True)
        t1 = time.perf_counter()
        s.prepare(div)
        s.set_vec("x", np.zeros((s.ny + 2, s.nz + 2, s.nx + 2)))
        s.set_tolerance(TOL)
        t2 = time.perf_counter()
        s.bicgstab(sample_iters)
        t3 = time.perf_counter()
        s.updated_winds(case.adv_den, u, v, w)
        t4 = time.perf_counter()
        t_iter = (t3 - t2) / sample_iters
        t_solve = (t1 - t0) + (t2 - t1) + (t4 - t3) + t_iter * ref_iters
        return {"value": 1.0 / t_solve, "t_iter_s": t_iter, "t_solve_s": t_solve, "t_sample_s": t4 - t0,
                "cores": self.cores, "extrapolated": True,
                "sample": f"divergence + RHS/diagonal + {sample_iters} of {ref_iters} BiCGStab iterations + "
                          f"lambda->winds timed; solve time extrapolated to {ref_iters} iterations "
                          f"(the count this method needs on this case)"}


def cpu_c1_baseline(repeats: int = 3) -> dict:
    """The primary CPU configuration (64x64x20, dx 250 m, 20 hills, alpha 1,
    density advected), timed in full: one steady-state solve (divergence,
    calc_iter_winds with the probed operator to 1e-6 from lambda = 0, wind
    correction) on all host cores and on one core, the iterations counted by
    the CPU solve itself.  Median of `repeats` solves each."""
    import numpy as np
    from oracle import oracle as O
    O.build()
    wl = WORKLOADS["cpu64"]
    case = build_inputs(wl, seed=1)
    s = O.OracleSolver(case.domain, "ref")
    s.set_alpha(case.alpha)
    u, v, w = (np.ascontiguousarray(a).copy() for a in (case.u, case.v, case.w))
    s.build_analytic(case.alpha)
    s.calibrate(case.adv_den, u, v, w)
    s.set_tolerance(TOL)
    all_cores = O.lib("ref").orc_get_threads()
    out = {"workload": "cpu64: 64x64x20 terrain case, 20 hills, alpha=const, adv_den=True", "tol_rel": TOL,
           "method": "BiCGStab + 2-sweep Jacobi-Richardson, probed operator, FP64 Krylov (the oracle)"}
    for tag, threads in (("all_cores", all_cores), ("1core", 1)):
        O.set_threads(threads)
        times, iters = [], None
        for _ in range(repeats):
            u, v, w = (np.ascontiguousarray(a).copy() for a in (case.u, case.v, case.w))
            s.set_vec("x", np.zeros((s.ny + 2, s.nz + 2, s.nx + 2)))
            t0 = time.perf_counter()
            div = s.divergence(u, v, w, adv_den=True)
            rc, st = s.calc_iter_winds(case.alpha, div, case.adv_den, u, v, w)
            times.append(time.perf_counter() - t0)
            iters = st["iters"]
            assert rc == 0 and st["status"] == 0, st
        out[f"solves_per_s_{tag}"] = 1.0 / statistics.median(times)
        out[f"cores_{tag}"] = threads
        out["iterations"] = iters
    O.set_threads(all_cores)
    s.close()
    return out


def workload_name(args, wl) -> str:
    """The workload as both arms name it in their JSON lines."""
    return (f"{args.workload}: {wl['nx']}x{wl['ny']}x{wl['nz']} terrain case, {wl['n_hills']} hills, "
            f"alpha={wl['alpha']}, adv_den={wl['adv_den']}")


def run_reference(args, wl):
    rank, world, local = dist_setup()
    if rank != 0:
        return
    case = build_inputs(wl, seed=1)
    cs = CpuSample(case)
    vals, samples, info = [], [], None
    for q in range(args.warmup + args.steps):
        info = cs.run(args.ref_iters, args.cpu_sample_iters)
        if q >= args.warmup:
            vals.append(info["value"])
            samples.append(info["t_sample_s"])
    v = statistics.median(vals)
    c1 = None if args.no_cpu_c1 else cpu_c1_baseline()
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup,
            # each timed step is the bounded CPU sample; value is the solve rate extrapolated from it
            "ms_per_step": 1000.0 * statistics.mean(samples), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": workload_name(args, wl), "tol_rel": TOL, "fields": "f32",
                       "method": "BiCGStab + 2-sweep Jacobi-Richardson, probed operator (the reference's "
                                 "method, restated on the CPU)",
                       "extrapolated": True, "ref_iters": args.ref_iters,
                       "ref_iters_source": REF_ITERS_SOURCE.get(args.workload, "command line"),
                       "ms_per_solve_extrapolated": 1000.0 / v,
                       "l2": "inputs larger than L2", "parallelism": "host cores"},
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": info["cores"], "kind": "port",
                             "sample": info["sample"], "extrapolated": True},
            "cpu_baseline_c1": c1,
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


# --------------------------------------------------------------------------------------
# GPU arm
# --------------------------------------------------------------------------------------
def profile_roofline(lib, h, stream, ncu_range: bool, cells: int, fp64_vectors: bool = True):
    """Per-launch CUDA-event profile of one solve iteration of handle h (every
    kernel of the iteration launched on its own, timed on `stream`) -> the
    roofline object of the dominant kernel."""
    import ctypes as C

    import torch
    cap = 32
    names = C.create_string_buffer(32 * cap)
    ms = (C.c_double * cap)()
    by = (C.c_double * cap)()
    cnt = (C.c_int * cap)()
    # one untimed pass first: the first launches of a kernel can carry one-time costs
    lib.hicarw_profile_iteration(h, 1, names, ms, by, cnt, cap, stream.cuda_stream)
    if ncu_range:
        torch.cuda.synchronize()
        torch.cuda.cudart().cudaProfilerStart()
    n = lib.hicarw_profile_iteration(h, 5, names, ms, by, cnt, cap, stream.cuda_stream)
    if ncu_range:
        torch.cuda.cudart().cudaProfilerStop()
    prof = []
    for q in range(max(n, 0)):
        nm = names.raw[32 * q:32 * q + 32].split(b"\0")[0].decode()
        prof.append({"kernel": nm, "ms": ms[q], "bytes": by[q], "per_iter": cnt[q], "share_ms": ms[q] * cnt[q]})
    if not prof:
        return None
    tot = sum(p["share_ms"] for p in prof) or 1.0
    dom_k = max(prof, key=lambda p: p["share_ms"])
    peak, peak_kind = peaks()
    ach = dom_k["bytes"] / (dom_k["ms"] * 1e-3) / 1e9
    return {"bound": "hbm", "kernel": dom_k["kernel"], "achieved": ach, "peak": peak, "unit": "GB/s",
            "frac": ach / peak, "peak_kind": peak_kind,
            "traffic": (TRAFFIC_PER_CELL[(dom_k["kernel"], fp64_vectors)] * cells
                        if (dom_k["kernel"], fp64_vectors) in TRAFFIC_PER_CELL else None),
            "share": dom_k["share_ms"] / tot,
            "kernels": [{k: (round(v, 6) if isinstance(v, float) else v) for k, v in p.items()} for p in prof]}


class OracleCheck:
    """The CPU oracle (reference precision) on the bench's case, outside every
    timed region: the GPU's probed operator (bit-exact with the oracle's own
    27-colour calibration, tests/test_gpu_parity.py), the oracle's own
    divergence of the input winds and its right-hand side (compute_rhs_3d).
    It certifies a GPU solution by the oracle's FP64 residual |b - A lambda| /
    |b| and corrects the input winds with the oracle's calc_updated_winds of
    that solution (wind_iterative.F90:1742-2071)."""

    def __init__(self, case, coefs):
        import numpy as np
        from oracle import oracle as O
        O.build()
        self.np, self.case = np, case
        self.s = O.OracleSolver(case.domain, "ref")
        self.s.set_alpha(case.alpha)
        self.s.set_coefs(coefs, probed=True)
        u, v, w = self.winds_in()
        self.div = self.s.divergence(u, v, w, adv_den=case.adv_den)
        self.div_norm = float(np.linalg.norm(self.div.astype(np.float64)))
        self.s.prepare(self.div)
        self.b_norm = float(np.linalg.norm(self.s.vec("rhs")))

    def winds_in(self):
        return tuple(self.np.ascontiguousarray(a).copy() for a in (self.case.u, self.case.v, self.case.w))

    def certify(self, lam):
        """(FP64 true residual of lam relative to |b|, corrected winds, final divergence relative to the input's)."""
        np, s = self.np, self.s
        s.set_vec("x", lam)
        res = s.true_residual() / self.b_norm
        u, v, w = self.winds_in()
        s.updated_winds(self.case.adv_den, u, v, w)
        d2 = s.divergence(u, v, w, adv_den=self.case.adv_den)
        return res, (u, v, w), float(np.linalg.norm(d2.astype(np.float64))) / self.div_norm

    def close(self):
        self.s.close()


def accuracy_report(lib, wi, wind, dom, h, div, u0, v0, w0, wl, stream, opts, tols, oracle_check):
    """Relative L2 differences of lambda and u/v/w between a solve with the
    timed options at each tolerance of `tols` and the converged solution, and
    the final divergence of the corrected winds relative to the input's.  The
    converged solution is a tight FP64 GPU solve (FGMRES + V-cycle to 1e-11)
    certified by the CPU oracle: its FP64 residual in the oracle's operator,
    and the reference winds are the oracle's correction of that lambda.
    Returns the report and compare(): the same differences for the solution
    and corrected winds the handle and domain hold after any later solve of
    the workload."""
    import torch
    from hicar_b200 import _capi

    def state():
        lam = torch.empty((dom.ny + 2, dom.nz + 2, dom.nx + 2), dtype=torch.float64, device=div.device)
        lib.hicarw_get_lambda(h, lam.data_ptr(), _capi.MEM_DEVICE, stream.cuda_stream)
        winds = [a.clone() for a in (dom.u_dqdt, dom.v_dqdt, dom.w_dqdt)]
        wind.calc_divergence(div, dom, use_dqdt=True)
        return lam, winds, float(div.double().norm())

    def solve_with(opt):
        wi.set_options(opt)
        dom.set_winds(u0, v0, w0)
        lib.hicarw_reset_solution(h, stream.cuda_stream)
        wind.calc_divergence(div, dom, use_dqdt=True)
        st = wi.calc_iter_winds(dom, dom.wind_alpha, div, wl["adv_den"])
        return (st,) + state()

    dom.set_winds(u0, v0, w0)
    wind.calc_divergence(div, dom, use_dqdt=True)
    d0 = float(div.double().norm())
    tight = solver_options("fgmres")
    tight.tol_rel, tight.wind_solver_iterations, tight.stall_iters = 1e-11, 6000, 0
    st_t, lam_t, _, _ = solve_with(tight)
    res_t, w_ref, div_ref = oracle_check.certify(lam_t.cpu().numpy())
    w_ref = [torch.from_numpy(a).to(div.device) for a in w_ref]

    def rel(a, b):
        return float((a.double() - b.double()).norm() / b.double().norm())

    def errors(lam, w_a, dn):
        return {"lambda_rel_l2": rel(lam, lam_t), "u_rel_l2": rel(w_a[0], w_ref[0]), "v_rel_l2": rel(w_a[1], w_ref[1]),
                "w_rel_l2": rel(w_a[2], w_ref[2]), "final_div_rel": dn / d0}

    def compare():
        return errors(*state())

    out = {"reference_solve": "FP64 FGMRES(30) + V-cycle to 1e-11 on the GPU, certified by the CPU oracle's FP64 "
                              "residual; winds from the oracle's calc_updated_winds of that lambda",
           "reference_iterations": st_t["iterations"], "reference_oracle_true_res_rel": res_t,
           "final_div_rel_reference": div_ref}
    for tol in tols:
        st, lam, w_a, dn = solve_with(at_tolerance(opts, tol))
        out[f"{tol:g}"] = {"iterations": st["iterations"], **errors(lam, w_a, dn)}
    return out, compare


def dataclasses_asdict(opt) -> dict:
    import dataclasses
    return {f.name: getattr(opt, f.name) for f in dataclasses.fields(opt)}


def at_tolerance(opt, tol):
    """`opt` at the relative tolerance `tol`.  FP32 Krylov vectors stagnate near
    3e-8 relative residual, so below 1e-7 the solve also stops on the FP64 true
    residual and restarts from it (iterative refinement, HICARW_CRIT_TRUE)."""
    from hicar_b200 import _capi, wind_iterative as wi
    kw = {**dataclasses_asdict(opt), "tol_rel": tol}
    if int(opt.krylov_precision) == _capi.KRYLOV_F32_X64 and tol < 1e-7:
        kw["criterion"] = _capi.CRIT_TRUE
    return wi.WindOptions(**kw)


def learned_report(lib, wi, dom, h, step, stream, tols, plain_ms, accuracy_solve=None):
    """The learned+mixed solver on the workload: FGMRES(30) with the composite
    preconditioner z = M(r) + theta U(r'), r' = r - A M(r), theta the
    minimal-residual step (the benchmark's V-cycle, then the
    U-Net trained on solver-logged pairs of 128x128x32 terrains, BF16 tensor-core
    convolutions), against the same outer loop with the V-cycle alone (the
    method without the network).  For each tolerance: solves/s of 3 timed
    solves (after one untimed), iterations, and the speed-up over the plain GPU
    BiCGStab.  None when no trained parameters are shipped."""
    import torch
    from hicar_b200 import _capi, learned as L
    from hicar_b200.train_unet import COMPOSITE_WEIGHTS, load_params
    if not os.path.exists(COMPOSITE_WEIGHTS):
        return None
    net = L.UNet(dom.nx, dom.ny, dom.nz)
    net.set_params(torch.from_numpy(load_params(COMPOSITE_WEIGHTS)))
    net.attach(h)
    out = {"weights": os.path.relpath(COMPOSITE_WEIGHTS, ROOT)}
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for tol in tols:
        for tag, pre in (("learned", _capi.PRECOND_MG_LEARNED), ("fgmres_mg", _capi.PRECOND_MG)):
            wi.set_options(wi.WindOptions(tol_rel=tol, wind_solver_iterations=3000, solver=_capi.SOLVER_FGMRES,
                                          precond=pre, fgmres_restart=30, stall_iters=200, **L.MG_CYCLE))
            step()
            torch.cuda.synchronize()
            e0.record()
            sts = [step() for _ in range(3)]
            e1.record()
            torch.cuda.synchronize()
            v = 3.0 / (e0.elapsed_time(e1) / 1000.0)
            key = f"{tag}_{tol:g}"
            out[key] = {"solves_per_s": v, "iterations": sts[0]["iterations"], "status": sts[0]["status"],
                        "precond": sts[0]["precond"], "true_res_rel": sts[0]["true_res"] / sts[0]["b_norm"],
                        "speedup_vs_plain_gpu": v / (1000.0 / plain_ms)}
            if accuracy_solve is not None and tag == "learned":
                out[key].update(accuracy_solve())
    lib.hicarw_set_learned_precond(h, None)
    net.close()
    # the U-Net's full-resolution 16 -> 16 convolution on this grid, against the
    # tensor-core and HBM rooflines (the Krylov part's bytes are the V-cycle's)
    c = L.conv_benchmark(16, 16, dom.nx, dom.ny, dom.nz, reps=5)
    tc_peak = bf16_sustained()
    hbm, _ = peaks()
    out["conv16"] = {**c, "tflops_frac_of_sustained_bf16": c["tflops"] / tc_peak if tc_peak else None,
                     "hbm_frac": c["gbs"] / hbm}
    return out


def run_ours(args, wl):
    import ctypes as C

    import numpy as np
    import torch
    from hicar_b200 import _capi, wind, wind_iterative as wi
    from hicar_b200.domain import DeviceDomain

    rank, world, local = dist_setup()
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    lib = _capi.load()
    case = build_inputs(wl, seed=subdomain_seed(rank))
    dom = DeviceDomain.from_case(case, f"cuda:{local}")
    u0, v0, w0 = dom.u_dqdt.clone(), dom.v_dqdt.clone(), dom.w_dqdt.clone()
    stream = torch.cuda.current_stream()
    wi.set_stream(stream.cuda_stream)
    opt0 = wi.WindOptions(advect_density=wl["adv_den"])
    wi.init_iter_winds(dom, opt0)
    div = torch.empty((dom.ny, dom.nz, dom.nx), dtype=torch.float32, device=f"cuda:{local}")
    wind.update_winds_iterative(dom, opt0, div)          # analytic solve + calibration + polish (untimed)
    h = wi.handle(dom.nest_indx)
    # iterations the reference method needs on this system (for the CPU extrapolation)
    opt = solver_options("plain")
    wi.set_options(opt)
    dom.set_winds(u0, v0, w0)
    lib.hicarw_reset_solution(h, stream.cuda_stream)
    wind.calc_divergence(div, dom, use_dqdt=True)
    p0, p1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    p0.record()
    ref_stats = wi.calc_iter_winds(dom, dom.wind_alpha, div, wl["adv_den"])
    p1.record()
    torch.cuda.synchronize()
    plain_ms = p0.elapsed_time(p1)  # one plain GPU BiCGStab solve (reference method), for the speed-up
    ref_iters = ref_stats["iterations"]
    opt = solver_options(args.solver)
    wi.set_options(opt)
    net = None
    if args.solver == "learned":  # trained parameters, shipped with the package
        from hicar_b200 import learned as L
        from hicar_b200.train_unet import load_params
        net = L.UNet(dom.nx, dom.ny, dom.nz)
        net.set_params(torch.from_numpy(load_params()))
        net.attach(h)

    def step():
        dom.set_winds(u0, v0, w0)
        lib.hicarw_reset_solution(h, stream.cuda_stream)
        wind.calc_divergence(div, dom, use_dqdt=True)
        return wi.calc_iter_winds(dom, dom.wind_alpha, div, wl["adv_den"])

    cycle = None
    if args.solver == "mg":
        overridden = MG_COARSE_SCALE is not None or MG_OMEGA is not None or MG_SKIP_FINE_PRE or bool(MG_W_LEVELS)
        if MG_CYCLE == "auto" and not overridden:
            opt, name, table = pick_cycle(wi, step, solver_kwargs(args.solver))
            cycle = {"chosen": name, "warmup_solve_ms": table, **MG_CYCLES[name.split("/")[0]]}
        elif MG_CYCLE != "auto":
            extra = {}
            if args.krylov_precision is not None:
                extra["krylov_precision"] = args.krylov_precision
            if args.mg_precision is not None:
                extra["mg_precision"] = args.mg_precision
            if MG_OMEGA is not None:  # the command line's smoother damping over the cycle's
                extra["mg_omega"] = MG_OMEGA
            opt = wi.WindOptions(**{**solver_kwargs(args.solver), **MG_CYCLES[MG_CYCLE], **extra})
            wi.set_options(opt)
            cycle = {"chosen": MG_CYCLE, **MG_CYCLES[MG_CYCLE], **extra}
        if cycle is not None:
            cycle = {k: (list(v) if isinstance(v, tuple) else v) for k, v in cycle.items()}
    if args.spmv_levels:  # z-march depth of the operator kernels (measurement; results do not depend on it)
        _capi.check(lib.hicarw_set_kernel_tuning(h, args.spmv_levels, -1), h)
    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    sampler = ClockSampler(local)
    sampler.start()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    l0 = lib.hicarw_kernel_launches()
    torch.cuda.synchronize()
    e0.record()
    stats = []
    for q in range(args.steps):
        if q == 0 and args.ncu_range == "step":
            torch.cuda.cudart().cudaProfilerStart()
        stats.append(step())
        if q == 0 and args.ncu_range == "step":
            torch.cuda.cudart().cudaProfilerStop()
    e1.record()
    torch.cuda.synchronize()
    launches = lib.hicarw_kernel_launches() - l0
    clocks = sampler.stop()
    t_ms = e0.elapsed_time(e1)
    t_ms = reduce_max(t_ms, dist, f"cuda:{local}")
    value = world * args.steps / (t_ms / 1000.0)

    # ---- e2e: the same step with host (pinned) winds copied in and out every step ----
    # Every step's input winds go host -> device and its corrected winds device ->
    # host inside the timed region, on a copy stream that overlaps them with the
    # neighbouring steps' solves (two device slots: the upload of step k + 1 and
    # the download of step k - 1 run while step k solves); only the first upload
    # and the last download are exposed.
    hu, hv, hw_ = (torch.empty(a.shape, dtype=torch.float32, pin_memory=True) for a in (u0, v0, w0))
    for src, dst in ((u0, hu), (v0, hv), (w0, hw_)):
        dst.copy_(src.cpu())
    # pinned results too (empty_like would not pin them): a device -> pageable copy blocks the host
    ou, ov, ow = (torch.empty(a.shape, dtype=torch.float32, pin_memory=True) for a in (hu, hv, hw_))
    h2d = sum(a.numel() * 4 for a in (hu, hv, hw_))
    d2h = h2d
    cstream = torch.cuda.Stream(device=f"cuda:{local}")
    slot_in = [tuple(torch.empty_like(a) for a in (u0, v0, w0)) for _ in range(2)]
    slot_out = [tuple(torch.empty_like(a) for a in (u0, v0, w0)) for _ in range(2)]
    up_done = [torch.cuda.Event() for _ in range(2)]
    solved = [torch.cuda.Event() for _ in range(2)]
    down_done = [None, None]  # the download that last read each output slot

    def upload(slot):
        with torch.cuda.stream(cstream):
            for dst, src in zip(slot_in[slot], (hu, hv, hw_)):
                dst.copy_(src, non_blocking=True)
            up_done[slot].record(cstream)

    def download(slot):
        with torch.cuda.stream(cstream):
            cstream.wait_event(solved[slot])
            for dst, src in zip((ou, ov, ow), slot_out[slot]):
                dst.copy_(src, non_blocking=True)
            down_done[slot] = torch.cuda.Event()
            down_done[slot].record(cstream)

    def e2e_run(n):
        down_done[0] = down_done[1] = None
        upload(0)
        st = None
        for k in range(n):
            q = k % 2
            if k + 1 < n:
                upload(1 - q)   # the slot step k - 1 read: its solve has returned
            if k > 0:
                download(1 - q)
            stream.wait_event(up_done[q])
            for dst, src in zip((dom.u_dqdt, dom.v_dqdt, dom.w_dqdt), slot_in[q]):
                dst.copy_(src)
            lib.hicarw_reset_solution(h, stream.cuda_stream)
            wind.calc_divergence(div, dom, use_dqdt=True)
            st = wi.calc_iter_winds(dom, dom.wind_alpha, div, wl["adv_den"])
            if down_done[q] is not None:
                stream.wait_event(down_done[q])  # the slot's previous results are on the host
            for dst, src in zip(slot_out[q], (dom.u_dqdt, dom.v_dqdt, dom.w_dqdt)):
                dst.copy_(src)
            solved[q].record(stream)
        download((n - 1) % 2)
        done = torch.cuda.Event()
        done.record(cstream)
        stream.wait_event(done)
        return st

    e2e_steps = max(3, args.steps)
    e2e_run(2)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    e0.record()
    e2e_run(e2e_steps)
    e1.record()
    torch.cuda.synchronize()
    te = e0.elapsed_time(e1)
    te = reduce_max(te, dist, f"cuda:{local}")
    e2e_value = world * e2e_steps / (te / 1000.0)
    assert np.array_equal(ou.numpy()[:1], dom.u_dqdt[:1].cpu().numpy(), equal_nan=True), \
        "the downloaded winds are the last step's"

    # ---- dominant kernel: per-launch CUDA-event profile of one iteration ----
    roofline = profile_roofline(lib, h, stream, args.ncu_range == "profile", dom.nx * dom.ny * dom.nz,
                                fp64_vectors=int(opt.krylov_precision) == 0)

    # ---- the same solve at the parity tolerance (lambda within 1e-5 of the converged solution) ----
    par = None
    if args.parity_tol and args.parity_tol != TOL:
        wi.set_options(at_tolerance(opt, args.parity_tol))
        step()
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        par_steps = max(1, min(args.steps, 5))
        e0.record()
        par_stats = [step() for _ in range(par_steps)]
        e1.record()
        torch.cuda.synchronize()
        tp = reduce_max(e0.elapsed_time(e1), dist, f"cuda:{local}")
        par = {"tol": args.parity_tol, "solves_per_s": world * par_steps / (tp / 1000.0),
               "iterations": par_stats[0]["iterations"],
               "true_res_rel": max(s_["true_res"] / s_["b_norm"] for s_ in par_stats)}
        wi.set_options(opt)

    # ---- accuracy against the converged solution, certified by the CPU oracle (rank 0, one GPU) ----
    accuracy, ocheck = None, None
    coefs = None
    if rank == 0 and world == 1 and not (args.no_accuracy and args.no_cpu):
        coefs = np.empty((15, dom.ny, dom.nz, dom.nx), np.float32)
        lib.hicarw_get_coefs(h, coefs.ctypes.data, _capi.MEM_HOST, stream.cuda_stream)
        ocheck = OracleCheck(case, coefs)
    compare = None
    if ocheck is not None and not args.no_accuracy:
        tols = [TOL] + ([args.parity_tol] if par else [])
        accuracy, compare = accuracy_report(lib, wi, wind, dom, h, div, u0, v0, w0, wl, stream, opt, tols, ocheck)
        wi.set_options(opt)

    # ---- the learned+mixed solver (FGMRES + V-cycle + U-Net correction) against FGMRES + V-cycle ----
    learned = None
    if world == 1 and not args.no_learned and args.solver == "mg":
        learned = learned_report(lib, wi, dom, h, step, stream, [TOL] + ([args.parity_tol] if par else []), plain_ms,
                                 compare)
        wi.set_options(opt)

    cpu = None
    if ocheck is not None and not args.no_cpu:
        c = CpuSample(case, solver=ocheck.s).run(ref_iters, args.cpu_sample_iters)
        cpu = {"value": c["value"], "unit": UNIT, "cores": c["cores"], "kind": "port", "sample": c["sample"],
               "t_iter_s": c["t_iter_s"], "extrapolated": True,
               "ref_iters_source": "the same method run to convergence on the GPU on this case"}
    if ocheck is not None:
        ocheck.close()
    c1 = cpu_c1_baseline() if rank == 0 and world == 1 and not (args.no_cpu or args.no_cpu_c1) else None

    it = [s["iterations"] for s in stats]
    tr = [s["true_res"] / s["b_norm"] for s in stats]
    acc_keys = {}
    if accuracy:
        for tag, tol in (("", TOL), ("parity_", args.parity_tol)):
            a_ = accuracy.get(f"{tol:g}")
            if a_:
                for k in ("lambda_rel_l2", "u_rel_l2", "v_rel_l2", "w_rel_l2", "final_div_rel"):
                    acc_keys[tag + k] = a_[k]
        acc_keys["final_div_rel_converged"] = accuracy["final_div_rel_reference"]
        acc_keys["converged_oracle_true_res_rel"] = accuracy["reference_oracle_true_res_rel"]
    if learned:
        for tag, tol in (("", TOL), ("parity_", args.parity_tol)):
            for name in ("learned", "fgmres_mg"):
                r_ = learned.get(f"{name}_{tol:g}")
                if r_:
                    acc_keys[f"{tag}{name}_solves_per_s"] = r_["solves_per_s"]
                    acc_keys[f"{tag}{name}_iterations"] = r_["iterations"]
                    acc_keys[f"{tag}{name}_speedup_vs_plain_gpu"] = r_["speedup_vs_plain_gpu"]
                    if "lambda_rel_l2" in r_:
                        acc_keys[f"{tag}{name}_lambda_rel_l2"] = r_["lambda_rel_l2"]
        if learned.get("conv16"):
            acc_keys["learned_conv16_tflops"] = learned["conv16"]["tflops"]
            acc_keys["learned_conv16_frac_of_sustained_bf16"] = learned["conv16"]["tflops_frac_of_sustained_bf16"]
            acc_keys["learned_conv16_hbm_frac"] = learned["conv16"]["hbm_frac"]
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": t_ms / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": ("f64" if opt.krylov_precision == 0 else "f32+f64") + ("+bf16" if opt.mg_precision else ""),
            "data": "synthetic",
            "config": {"workload": workload_name(args, wl),
                       "solver": args.solver, "mg_cycle_name": (cycle or {}).get("chosen"), "mg_cycle": cycle,
                       "spmv_levels": args.spmv_levels or None,
                       "tol_rel": TOL, "fields": "f32", "krylov": krylov_desc(opt),
                       "preconditioner_precision": ("bf16 coefficients in the finest level's smoother, f32 elsewhere"
                                                    if opt.mg_precision else "f32"),
                       "iterations": it[0], "ref_method_iterations": ref_iters, "true_res_rel": max(tr),
                       "plain_gpu_solves_per_s": 1000.0 / plain_ms,
                       "speedup_vs_plain_gpu": value / world / (1000.0 / plain_ms),
                       **acc_keys,
                       "parity_tol": par["tol"] if par else None,
                       "parity_tol_solves_per_s": par["solves_per_s"] if par else None,
                       "parity_tol_iterations": par["iterations"] if par else None,
                       "parity_tol_speedup_vs_plain_gpu": (par["solves_per_s"] / world / (1000.0 / plain_ms)
                                                           if par else None),
                       "accuracy": accuracy, "learned_fgmres": learned,
                       "l2": "inputs larger than L2 (15 FP32 coefficient arrays, %.2f GB)"
                             % (15 * 4 * (dom.nx + 2) * (dom.ny + 2) * (dom.nz + 2) / 1e9),
                       "parallelism": f"{world} independent subdomains" if world > 1 else "1 GPU"},
            "roofline": roofline, "cpu_baseline": cpu, "cpu_baseline_c1": c1,
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
            "clocks": clocks, "gpu_launches": int(launches)}
    wi.finalize_iter_winds()
    if world == 1 and not args.no_batch and args.workload == "mixed1024":
        torch.cuda.synchronize()
        del dom, div, u0, v0, w0, case  # the headline workload's device memory goes back before the batch
        net = compare = None
        torch.cuda.empty_cache()
        try:
            b = batch_measure(args, WORKLOADS["batch96"], rank, world, dist, local, quick=True)
        except Exception as e:  # the headline line is printed all the same, with the reason
            b = None
            line["config"]["batch96_error"] = f"{type(e).__name__}: {e}"
    if world == 1 and not args.no_batch and args.workload == "mixed1024" and b is not None:
        c = b["config"]
        line["config"].update({"batch96_solves_per_s": b["value"], "batch96_e2e_solves_per_s": b["e2e"]["value"],
                               "batch96_sequential_solves_per_s": c["sequential_solves_per_s"],
                               "batch96_p50_ms": c["batched_p50_ms"], "batch96_p99_ms": c["batched_p99_ms"],
                               "batch96_learned_subdomains": c["learned_subdomains"],
                               "batch96_iterations_max": c["iterations_max"]})
        line["batch96"] = {k: b[k] for k in ("value", "ms_per_step", "steps", "warmup", "config", "e2e", "clocks",
                                             "gpu_launches")}
    if rank == 0:
        print_line(line)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def batch_measure(args, wl, rank, world, dist, local, quick=False):
    """The batch workload: every step solves all subdomains (divergence, the
    batched solve in one graph launch, wind correction).  Three of every four
    subdomains use BiCGStab with the V-cycle, every fourth FGMRES with the
    composite learned preconditioner when trained parameters are shipped.  The
    kernel autotuner picks the operator kernels' z-march depth and the
    smoother's feed per subdomain-size bucket (quick: a reduced search), the
    batch autotuner the concurrent chains and iterations per loop body.
    Returns the JSON line."""
    import ctypes as C

    import numpy as np
    import torch
    from hicar_b200 import _capi
    from hicar_b200.batch import LEARNED_RESTART, BatchSolver, subdomain_cases
    from hicar_b200.domain import ptr
    from hicar_b200.train_unet import COMPOSITE_WEIGHTS, load_params
    from hicar_b200.wind_iterative import WindOptions

    lib = _capi.load()
    stream = torch.cuda.current_stream()
    cyc = MG_CYCLE if MG_CYCLE != "auto" else "V01-W24"  # batches: the cycle named on the command line
    opts = WindOptions(tol_rel=TOL, wind_solver_iterations=3000, precond=_capi.PRECOND_MG, stall_iters=50,
                       advect_density=wl["adv_den"], **MG_CYCLES[cyc])
    params = None
    if args.batch_learned_every > 0 and os.path.exists(COMPOSITE_WEIGHTS):
        params = torch.from_numpy(load_params(COMPOSITE_WEIGHTS))
    bs = BatchSolver(subdomain_cases(wl["batch"], seed=subdomain_seed(rank), nxy=wl["nxy"], nz=wl["nz"],
                                     n_hills=wl["n_hills"], dx=wl["dx"]), options=opts, stream=stream.cuda_stream,
                     learned_every=args.batch_learned_every if params is not None else 0, learned_params=params)
    try:
        kt = bs.autotune_kernels(levels=(16, 32) if quick else (8, 16, 32, 64), feeds=(1,) if quick else (1, 0))
        tuned_ms = bs.autotune()
        lanes, chunk = bs.config()
        # the same subdomains one after another through hicarw_calc_iter_winds (untimed by the contract; reported)
        bs.restore_winds()
        bs.divergence()
        torch.cuda.synchronize()
        q0, q1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        q0.record()
        st = _capi.Stats()
        seq_each = []
        for i, (h, dom) in enumerate(zip(bs.handles, bs.domains)):
            lib.hicarw_reset_solution(h, C.c_void_p(bs.stream))
            _capi.check(lib.hicarw_calc_iter_winds(h, ptr(dom.wind_alpha), ptr(bs.divs[i]), ptr(dom.density), 1,
                                                   ptr(dom.u_dqdt), ptr(dom.v_dqdt), ptr(dom.w_dqdt),
                                                   _capi.MEM_DEVICE, C.c_void_p(bs.stream), C.byref(st)), h)
            seq_each.append(st.solve_ms)
        q1.record()
        torch.cuda.synchronize()
        seq_ms = q0.elapsed_time(q1)
        steps, warmup = (3, 1) if quick else (args.steps, args.warmup)
        for _ in range(warmup):
            bs.step()
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        sampler = ClockSampler(local)
        sampler.start()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        l0 = lib.hicarw_kernel_launches()
        torch.cuda.synchronize()
        e0.record()
        stats = []
        for _ in range(steps):
            stats = bs.step()
        e1.record()
        torch.cuda.synchronize()
        launches = lib.hicarw_kernel_launches() - l0
        clocks = sampler.stop()
        t_ms = reduce_max(e0.elapsed_time(e1), dist, f"cuda:{local}")
        value = world * steps * bs.n / (t_ms / 1000.0)
        # e2e: every subdomain's winds from pinned host memory in, corrected winds out
        host = [[torch.empty(a.shape, dtype=torch.float32, pin_memory=True) for a in sv] for sv in bs.saved]
        for hs, sv in zip(host, bs.saved):
            for dst, src in zip(hs, sv):
                dst.copy_(src.cpu())
        outs = [[torch.empty(a.shape, dtype=torch.float32, pin_memory=True) for a in hs] for hs in host]
        h2d = sum(a.numel() * 4 for hs in host for a in hs)

        def e2e_step():
            for dom, hs in zip(bs.domains, host):
                dom.u_dqdt.copy_(hs[0], non_blocking=True)
                dom.v_dqdt.copy_(hs[1], non_blocking=True)
                dom.w_dqdt.copy_(hs[2], non_blocking=True)
            bs.divergence()
            bs.solve(cold=True)
            for dom, os_ in zip(bs.domains, outs):
                os_[0].copy_(dom.u_dqdt, non_blocking=True)
                os_[1].copy_(dom.v_dqdt, non_blocking=True)
                os_[2].copy_(dom.w_dqdt, non_blocking=True)

        e2e_step()
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        e0.record()
        e2e_steps = max(1, min(steps, 3))
        for _ in range(e2e_steps):
            e2e_step()
        e1.record()
        torch.cuda.synchronize()
        te = reduce_max(e0.elapsed_time(e1), dist, f"cuda:{local}")
        e2e_value = world * e2e_steps * bs.n / (te / 1000.0)
        big = max(range(bs.n), key=lambda i: bs.domains[i].nx * bs.domains[i].ny * bs.domains[i].nz)
        d_big = bs.domains[big]
        roofline = None if quick else profile_roofline(lib, bs.handles[big], stream, False,
                                                       d_big.nx * d_big.ny * d_big.nz)
        if roofline:
            roofline["profiled_subdomain"] = [d_big.nx, d_big.ny, d_big.nz]
        iters = [s_["iterations"] for s_ in stats]
        bs.step()
        lat = bs.latencies()
        seq_lat = np.asarray(seq_each)
        n_learned = sum(bs.learned)
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": steps,
                "warmup": warmup, "ms_per_step": t_ms / steps, "higher_is_better": True, "scaling": "weak",
                "vs_baseline": None, "dtype": "f64", "data": "synthetic",
                "config": {"workload": f"batch{bs.n}: {bs.n} subdomains, nx,ny in {wl['nxy'][0]}..{wl['nxy'][1]} "
                                       f"step {wl['nxy'][2]}, nz in {wl['nz'][0]}..{wl['nz'][1]} step {wl['nz'][2]}, "
                                       f"{bs.cells} cells, {wl['n_hills']} hills each, adv_den={wl['adv_den']}",
                           "solver": f"batched: BiCGStab + V-cycle ({bs.n - n_learned}), FGMRES({LEARNED_RESTART}) + "
                                     f"V-cycle + U-Net correction ({n_learned}); one graph launch per step",
                           "mg_cycle": cyc, "tol_rel": TOL, "fields": "f32", "krylov": "f64",
                           "lanes": lanes, "chunk": chunk, "autotune_best_ms": tuned_ms, "kernel_autotune": kt,
                           "learned_subdomains": n_learned,
                           "sequential_solves_per_s": bs.n / (seq_ms / 1000.0), "iterations_min": min(iters),
                           "iterations_max": max(iters), "statuses": sorted(set(s_["status"] for s_ in stats)),
                           "batched_p50_ms": float(np.percentile(lat, 50)),
                           "batched_p99_ms": float(np.percentile(lat, 99)), "batched_max_ms": float(lat.max()),
                           "sequential_p50_ms": float(np.percentile(seq_lat, 50)),
                           "sequential_p99_ms": float(np.percentile(seq_lat, 99)),
                           "latency_note": "batched: completion time of each solve from the start of the batch graph; "
                                           "sequential: each subdomain's own calc_iter_winds",
                           "l2": "inputs larger than L2 (coefficients of all subdomains)",
                           "parallelism": f"{world} ranks x {bs.n} subdomains" if world > 1 else "1 GPU"},
                "roofline": roofline, "cpu_baseline": None,
                "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": h2d},
                "clocks": clocks, "gpu_launches": int(launches)}
    finally:
        bs.close()
    return line


def run_batch(args, wl):
    """The batch workload as its own bench line."""
    import torch
    rank, world, local = dist_setup()
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))
    line = batch_measure(args, wl, rank, world, dist, local)
    if rank == 0:
        print_line(line)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def main():
    global TOL, MG_COARSE_SCALE, MG_OMEGA, MG_SKIP_FINE_PRE, MG_W_LEVELS, MG_CYCLE, FGMRES_RESTART
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="mixed1024", choices=sorted(WORKLOADS))
    ap.add_argument("--solver", default="mg", choices=["plain", "mg", "fgmres", "fgmres_jacobi", "learned"])
    ap.add_argument("--no-accuracy", action="store_true", help="skip the tight-solve accuracy report")
    ap.add_argument("--tol", type=float, default=TOL, help="relative residual tolerance of the timed solves")
    ap.add_argument("--mg-coarse-scale", type=float, default=None,
                    help="override the V-cycle's coarse-correction scale of the solver preset")
    ap.add_argument("--mg-skip-fine-presmooth", action="store_true",
                    help="V(0,1) on the finest level of the V-cycle (no pre-smoothing there)")
    ap.add_argument("--mg-cycle", default="auto", choices=["auto"] + list(MG_CYCLES),
                    help="cycle shape of the mg preset (auto: the fastest on the workload, picked in the warm-up)")
    ap.add_argument("--mg-w-levels", default="",
                    help="comma-separated V-cycle levels (>= 1) that correct twice from the coarse grid")
    ap.add_argument("--krylov-precision", type=int, default=None, choices=[0, 2],
                    help="with --mg-cycle NAME: Krylov vectors FP64 (0) or FP32 with FP64 lambda (2)")
    ap.add_argument("--mg-precision", type=int, default=None, choices=[0, 1],
                    help="with --mg-cycle NAME: finest-level smoother coefficients FP32 (0) or BF16 (1)")
    ap.add_argument("--mg-omega", type=float, default=None,
                    help="override the V-cycle's smoother damping of the solver preset")
    ap.add_argument("--fgmres-restart", type=int, default=None,
                    help="override the restart length of the FGMRES presets")
    ap.add_argument("--cpu-sample-iters", type=int, default=10)
    ap.add_argument("--ref-iters", type=int, default=None,
                    help="iterations of the reference method on the workload (reference arm)")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU oracle baselines")
    ap.add_argument("--no-cpu-c1", action="store_true", help="skip the full CPU solve of the 64x64x20 case")
    ap.add_argument("--batch-learned-every", type=int, default=4,
                    help="batch workloads: every m-th subdomain uses the learned preconditioner (0: none)")
    ap.add_argument("--no-batch", action="store_true",
                    help="skip the 96-subdomain batch measurement that the default run adds to its line")
    ap.add_argument("--no-learned", action="store_true",
                    help="skip the learned+mixed FGMRES report (run only when trained parameters are shipped)")
    ap.add_argument("--parity-tol", type=float, default=1e-9,
                    help="also time the solve at this tolerance and report its accuracy (0: off)")
    ap.add_argument("--spmv-levels", type=int, default=0,
                    help="levels per work item of the float4 operator kernels (0: the library's default)")
    ap.add_argument("--ncu-range", default="none", choices=["none", "step", "profile"],
                    help="bracket the first timed step or the per-kernel profiling pass with "
                         "cudaProfilerStart/Stop (for ncu --profile-from-start off)")
    args = ap.parse_args()
    TOL = args.tol
    MG_COARSE_SCALE = args.mg_coarse_scale
    MG_OMEGA = args.mg_omega
    MG_SKIP_FINE_PRE = args.mg_skip_fine_presmooth
    MG_W_LEVELS = tuple(int(x) for x in args.mg_w_levels.split(",") if x.strip())
    MG_CYCLE = args.mg_cycle
    FGMRES_RESTART = args.fgmres_restart
    wl = WORKLOADS[args.workload]
    if "batch" in wl:
        if args.impl == "reference":
            print(json.dumps({"impl": "reference", "unavailable": "the batch workload has no CPU reference arm; "
                                                                  "its subdomains are timed one by one on the GPU "
                                                                  "(config.sequential_solves_per_s)"}))
            return
        run_batch(args, wl)
        return
    if args.impl == "reference":
        if args.ref_iters is None:
            args.ref_iters = REF_ITERS[args.workload]
        run_reference(args, wl)
    else:
        run_ours(args, wl)


if __name__ == "__main__":
    main()
