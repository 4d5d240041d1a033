#!/usr/bin/env python
"""Benchmark of the AM sparse-PCA hot path (start-iterations per second).

Workload (one GPU): n = 2000 samples x p = 50000 features, low-rank (r = 50,
256 non-zeros per loading) plus N(0, 0.1^2) noise, seeded and generated on
the device; k = 1024 starting points U[-1, 1] normalised; all 8 formulations:
s = 16 for the constraint forms, gamma = 0.1 x max column 2-norm (L2-variance
penalties) or 0.1 x max column 1-norm (L1-variance penalties).  FP32 data;
tensor-core products FP32-accurate: 3xTF32 (L2-variance forms), or for the
L1-variance forms, whose Z = sgn(B V) is exact in BF16, B split exactly into
three BF16 planes; FP32 accumulation.

A step is one AM iteration of every formulation over its k starts, i.e.
8 x 1024 start-iterations.  `value` = start-iterations/s of the whole job with
the data resident in HBM (device-timed with CUDA events on the library's
stream, max over ranks).  `e2e` is the same metric through the public
one-call API am24_solve_dense_f32 with host (pinned) buffers, host<->device
copies included, each formulation solved to its own convergence (maxIter 200,
tol 1e-6).  `roofline` is for the dominant kernel, from per-kernel CUDA events
inside the timed steps.  `cpu_baseline` times the reference's own CPU solver
(built from its sources, multithreaded OpenBLAS) on a bounded sample.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Multi-GPU: one process per GPU under torchrun; every rank runs the same
workload on its own starting points (start sharding, weak scaling, no
collective on the data path).
"""
import argparse
import ctypes as C
import importlib
import json
import os
import re
import statistics
import subprocess
import sys
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

SIZES = {  # (n samples, p features, rank, nnz per loading, starts)
    "config1": (2000, 50000, 50, 256, 1024),
    # profiling case: same kernels, B planes 262 MB (> L2), a few GB on the device
    "small": (2000, 8192, 50, 256, 1024),
    # mixed-precision workload (whole solves, --mode solve): s = 128
    "config2": (8192, 65536, 100, 512, 4096),
}
SIZE_S = {"config1": 16, "small": 16, "config2": 128}
# gamma = factor x the largest column norm: at n = 8192 samples, 0.1 x the
# largest column 1-norm lies above every loading and empties every support
SIZE_GAMMA = {"config1": 0.1, "small": 0.1, "config2": 0.025}
N_SAMPLES, P_FEATURES, RANK, NNZ_V, STARTS = SIZES["config1"]
S_CONS, GAMMA_C, SEED = 16, 0.1, 1
E2E_MAX_IT, E2E_TOL = 200, 1e-6
CPU_SAMPLE_STARTS, CPU_SAMPLE_ITERS = 64, 3
CPU_SAMPLE_STARTS_PORT = 4  # the one-core port takes 0.65 s a start-iteration: a minute
def workload_name():
    tag = "config-1" if (N_SAMPLES, P_FEATURES) == SIZES["config1"][:2] else "profiling case"
    return (f"{tag} AM step: n={N_SAMPLES} samples x p={P_FEATURES} features (r={RANK}, "
            f"{NNZ_V} nnz/loading), k={STARTS} starts, 8 formulations, plain FP32 path")


def bench_config(world, forms):
    """The workload's description, the same on both arms."""
    return {"workload": workload_name(), "n": N_SAMPLES, "p": P_FEATURES,
            "starts_per_gpu": STARTS, "formulations": forms, "s": S_CONS,
            "gamma_factor": GAMMA_C, "precision": PRECISION_NOTE,
            "l2": "inputs larger than L2 (B as FP32 and two FP16 planes each way: 1.2 GB)",
            "parallelism": f"start-sharded x{world}, no data-path collective"}


def dist_env():
    return (int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)),
            int(os.environ.get("LOCAL_RANK", 0)))


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return d, "measured"
    except Exception:
        return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0}, \
            "fallback"


def profiled_traffic(kernel):
    """DRAM bytes per launch of `kernel` on this workload from the committed ncu
    summary (profiles/), or None."""
    path = os.path.join(ROOT, "profiles", "am_step_2000x50000_k1024.md")
    try:
        txt = open(path).read()
    except OSError:
        return None
    m = re.search(rf"^traffic_bytes_per_launch\s+{re.escape(kernel)}\s+([0-9.eE+]+)", txt, re.M)
    return float(m.group(1)) if m else None


class ClockSampler:
    """nvidia-smi clock / throttle samples during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu, period_ms=100):
        self.period = str(int(period_ms))
        vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
        ids = [v.strip() for v in vis.split(",") if v.strip()]
        self.gpu = ids[gpu] if gpu < len(ids) else str(gpu)
        self.p = None

    def __enter__(self):
        try:
            self.p = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", self.period],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.p = None
        return self

    def __exit__(self, *a):
        self.lines = []
        if self.p:
            self.p.terminate()
            try:
                out, _ = self.p.communicate(timeout=5)
            except Exception:
                self.p.kill()
                out, _ = self.p.communicate()
            self.lines = [l for l in out.splitlines() if l.strip()]

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in getattr(self, "lines", []):
            f = [x.strip() for x in l.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for name, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


# ------------------------------------------------------------------ CPU legs
def cpu_reference(B_host, steps, per_step_iters, starts, forms_per_step=8, first_step=0):
    """The reference's own denseDataSolver<float> (oracle/_ref, OpenBLAS,
    all host threads) on n x p = B_host, `starts` starting points,
    `per_step_iters` iterations; each step solves `forms_per_step` formulations
    (all 8, or the next ones in turn from step `first_step` on); returns
    (start-it/s, cores, kind, start-iterations, seconds)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import numpy as np
    import pyoracle as po
    cores = os.cpu_count() or 1
    kind = "reference"
    blas = "openblas"
    if not po.ref_available(blas):
        blas = "naive"
    if not po.ref_available(blas):
        kind = "port"
    gam = {}
    col2 = float(np.sqrt((B_host.astype(np.float64) ** 2).sum(0)).max())
    col1 = float(np.abs(B_host).sum(0, dtype=np.float64).max())
    gam = {4: GAMMA_C * col2, 6: GAMMA_C * col2, 5: GAMMA_C * col1, 7: GAMMA_C * col1}
    if kind == "reference":
        po.ref_set_threads(cores, blas)
    total_its, total_s = 0, 0.0
    for step in range(steps):
        forms = (range(8) if forms_per_step >= 8 else
                 [((first_step + step) * forms_per_step + i) % 8 for i in range(forms_per_step)])
        for f in forms:
            s = po.make_settings(f, constraint=S_CONS, penalty=gam.get(f, 0.0), tolerance=0.0,
                                 max_iter=per_step_iters, total_starts=starts, batch_size=starts)
            if kind == "reference":
                r = po.ref_solve(B_host, s, blas=blas)
                total_s += r["compute_time"]
            else:
                t0 = time.perf_counter()
                r = po.oracle_solve(B_host, s)
                total_s += time.perf_counter() - t0
                cores = 1
            total_its += starts * int(r["it"])
    return total_its / total_s, cores, kind, total_its, total_s


def cpu_sample(B_host):
    """cpu_reference on the bounded sample of the full matrix that fits the code at
    hand: the reference's where it was built, else this repository's port of it on one
    core.  Its results, the starts sampled and the name of the code that ran."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle as po
    if po.ref_available("openblas"):
        code = "reference denseDataSolver<float> + OpenBLAS"
    elif po.ref_available("naive"):
        code = "reference denseDataSolver<float> + plain C BLAS"
    else:
        code = "one-core C port of the reference's solver"
    starts = CPU_SAMPLE_STARTS_PORT if code.startswith("one-core") else CPU_SAMPLE_STARTS
    return (*cpu_reference(B_host, 1, CPU_SAMPLE_ITERS, starts), starts, code)


def fp64_oracle_check(am, M, B_host, gam, starts=64, iters=3):
    """Per-start error of the GPU path against the FP64 oracle (checker only,
    outside every timed region): for each formulation, `starts` reference
    starting points stepped `iters` times on the device (am24_batch_iterate)
    and by oracle/fast_oracle in FP64 from the same FP32 starts.  Returns, per
    formulation, the largest and median relative difference of the per-start
    objective and of the per-start explained variance ||B x||^2 (FP64 of each
    side's loadings), over the starts whose steps were all well conditioned,
    and how many were set aside."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import numpy as np
    import pyoracle as po
    import fast_oracle as fo
    B64 = np.asarray(B_host, np.float64)
    n = B64.shape[1]
    out = {}
    for f in range(8):
        V0 = po.reference_starts(n, starts, f <= 3, S_CONS, dtype=np.float32)
        st = am.OptimizationSettings(formulation=f, constraintParameter=S_CONS,
                                     penaltyParameter=gam.get(f, 0.0), tolerance=0.0,
                                     maximumIterations=iters, totalStartingPoints=starts,
                                     batchSize=starts)
        b = M.batch(st, starts)
        b.load(V0)
        b.iterate(0, iters)
        Vg, valg, _, _ = b.read()
        b.close()
        V = V0.astype(np.float64)
        val = np.zeros(starts)
        ill = np.zeros(starts, bool)
        for _ in range(iters):
            r = fo.iteration(B64, V, f, S_CONS, gam.get(f, 0.0), val)
            V, val, ill = r.V, r.val, ill | r.ill
        ok = ~ill & np.isfinite(val) & (val != 0)
        with np.errstate(divide="ignore", invalid="ignore"):
            e_obj = np.abs(valg.astype(np.float64) - val) / np.abs(val)

            def ev(X):
                Xn = X / np.linalg.norm(X, axis=0, keepdims=True)
                return np.linalg.norm(B64 @ Xn, axis=0) ** 2
            e_ev = np.abs(ev(Vg.astype(np.float64)) - ev(V)) / ev(V)
        o, v = e_obj[ok], e_ev[ok]
        out[str(f)] = {"max_objective_rel_err": float(o.max()) if o.size else None,
                       "median_objective_rel_err": float(np.median(o)) if o.size else None,
                       "max_explained_variance_rel_err": float(v.max()) if v.size else None,
                       "starts_compared": int(ok.sum()), "set_aside_ill_conditioned":
                           int(starts - ok.sum())}
    return out


def run_reference_arm(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return 0
    import numpy as np
    am = importlib.import_module("24am_b200")
    wl = am.workloads
    import torch
    if torch.cuda.is_available():
        B = wl.low_rank_data_torch(N_SAMPLES, P_FEATURES, RANK, NNZ_V, SEED).cpu().numpy()
    else:
        B = wl.low_rank_data(N_SAMPLES, P_FEATURES, RANK, NNZ_V, SEED, dtype=np.float32).T.copy()
    B_host = np.asfortranarray(B.T)  # n x p column-major
    # the GPU arm's configuration (all k starts of a batch, the full matrix);
    # each step one iteration of one formulation, the eight in turn, so that
    # the run stays within minutes
    cpu_reference(B_host, args.warmup, 1, STARTS, forms_per_step=1)  # untimed warm-up
    t0 = time.time()
    v, cores, kind, its, secs = cpu_reference(B_host, args.steps, 1, STARTS, forms_per_step=1,
                                              first_step=args.warmup)
    wall = time.time() - t0
    sample = (f"{args.steps} steps, each 1 iteration of one formulation (the 8 in turn) x "
              f"{STARTS} starts on the full {N_SAMPLES}x{P_FEATURES} matrix ({its} "
              f"start-iterations, {secs:.1f} s compute)")
    line = {"impl": "reference", "metric": "start-iterations/s", "value": v,
            "unit": "start-it/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * secs / max(args.steps, 1), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": bench_config(world, list(range(8))),
            "cpu_baseline": {"value": v, "unit": "start-it/s", "cores": cores, "kind": kind,
                             "sample": sample},
            "e2e": {"value": v, "unit": "start-it/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0},
            "wall_s": wall}
    print(json.dumps(line), flush=True)
    return 0


# ------------------------------------------------------------------ GPU arm
def run_solves(args):
    """Whole solves on one GPU (resident matrix, injected seeded starts, one batch
    of all starts, maxIter 200, tol 1e-6), each formulation in FP32 and in MIXED
    precision.  start-iterations/s from the library's CUDA-event time of the
    iterations; the best explained variance ||B x||^2 is evaluated in FP64 on the
    device, and the line gives MIXED's relative difference from FP32's."""
    import numpy as np
    import torch
    am = importlib.import_module("24am_b200")
    wl = am.workloads
    solver = am.Solver(0)
    Dt = wl.low_rank_data_torch(N_SAMPLES, P_FEATURES, RANK, NNZ_V, SEED)
    col2 = float(Dt.double().norm(dim=1).max())
    col1 = float(Dt.double().abs().sum(dim=1).max())
    gam = wl.penalty_gammas(col2, col1, GAMMA_C)
    torch.cuda.synchronize()
    M = am.Matrix(solver, None, on_device_ptr=Dt.data_ptr(), m=N_SAMPLES, n=P_FEATURES,
                  ldB=N_SAMPLES)
    forms = [int(x) for x in args.formulations.split(",")]
    res = {}
    tot = {"fp32": [0, 0.0], "mixed": [0, 0.0]}
    for f in forms:
        V = wl.uniform_starts_torch(P_FEATURES, STARTS, seed=1000 + SEED + f).cpu().numpy()
        V = np.asfortranarray(V.T)  # p x k column-major
        row = {}
        for name, prec in (("fp32", am.PRECISION_FP32), ("mixed", am.PRECISION_MIXED)):
            st = am.OptimizationSettings(formulation=f, constraintParameter=S_CONS,
                                         penaltyParameter=gam.get(f, 0.0), tolerance=E2E_TOL,
                                         maximumIterations=E2E_MAX_IT, totalStartingPoints=STARTS,
                                         batchSize=STARTS, startMode=am.START_INJECTED,
                                         precision=prec,
                                         leadIterations=args.mixed_lead if prec else 0)
            _, fval, s = M.solve(st, start_points=V)
            row[name] = {"start_it_per_s": s.start_iterations / s.total_true_computation_time,
                         "iterations": int(s.it), "bf16_iterations": int(s.low_precision_iterations),
                         "seconds": s.total_true_computation_time, "fval": fval,
                         "explained_variance": s.explained_variance}
            tot[name][0] += int(s.start_iterations)
            tot[name][1] += s.total_true_computation_time
        ev32, evmx = row["fp32"]["explained_variance"], row["mixed"]["explained_variance"]
        row["ev_rel_diff"] = abs(evmx - ev32) / ev32
        res[str(f)] = row
    v32 = tot["fp32"][0] / tot["fp32"][1]
    vmx = tot["mixed"][0] / tot["mixed"][1]
    line = {"metric": "start-iterations/s (whole solves to tol)", "value": vmx,
            "unit": "start-it/s", "n_gpus": 1, "higher_is_better": True, "dtype": "bf16+f32",
            "data": "synthetic",
            "config": {"workload": f"mixed precision solves: n={N_SAMPLES} x p={P_FEATURES} "
                                   f"(r={RANK}, {NNZ_V} nnz/loading), k={STARTS} starts, "
                                   f"s={S_CONS}, gamma {GAMMA_C} x max column norm, "
                                   f"formulations {forms}, maxIter {E2E_MAX_IT}, tol {E2E_TOL}",
                       "precision": (f"MIXED: {args.mixed_lead} FP32-accurate iterations, then "
                                     "single-pass FP16 V = B^T Z until every start's support is "
                                     "unchanged for 5 iterations, then FP32-accurate")},
            "fp32_value": v32, "speedup_vs_fp32": vmx / v32,
            "max_ev_rel_diff": max(r["ev_rel_diff"] for r in res.values()),
            "formulations": res}
    print(json.dumps(line), flush=True)
    M.close()
    solver.close()
    return 0


def config3_problems(am, count, matrices, seed):
    """Requests from the uneven-problem distribution: a resident matrix each,
    formulation uniform over the 8, s uniform in [8, 256], starts uniform in
    [32, 1024], gamma 0.1 x the matrix's largest column 2-norm (L2-variance
    penalties) or 0.025 x its largest column 1-norm (L1-variance penalties),
    maxIter 200, tol 1e-6, starting points U[-1, 1] normalised, generated on
    the device."""
    import numpy as np
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        mid, m, n, c2, c1 = matrices[int(rng.integers(len(matrices)))]
        f = int(rng.integers(8))
        st = am.OptimizationSettings(
            formulation=f, constraintParameter=int(rng.integers(8, 257)),
            penaltyParameter=(0.1 * c2 if f in (4, 6) else 0.025 * c1),
            tolerance=1e-6, maximumIterations=200,
            totalStartingPoints=int(rng.integers(32, 1025)), batchSize=0,
            startMode=am.START_DEVICE_UNIFORM)
        out.append((mid, n, st))
    return out


def uneven_problems(am, wl, count, seed):
    """The uneven-problem workload: `count` independent problems, each on its
    own matrix from the low-rank-plus-noise generator (n log-uniform in
    [100, 5000] samples, p log-uniform in [1e3, 1e5] features,
    r = min(n, p) / 20, 64 non-zeros per loading), its own formulation
    (uniform over the 8), s uniform in [8, 256], starts uniform in [32, 1024]
    (U[-1, 1] normalised, generated on the device), gamma 0.1 x the matrix's
    largest column 2-norm (L2-variance penalties) or 0.025 x its largest column
    1-norm (L1-variance penalties), maxIter 200, tol 1e-6.  Yields
    (m, n, seed, settings kwargs) per problem; matrices are generated on demand."""
    import numpy as np
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        n = int(np.exp(rng.uniform(np.log(100), np.log(5000))))
        p = int(np.exp(rng.uniform(np.log(1000), np.log(100000))))
        f = int(rng.integers(8))
        s = int(rng.integers(8, 257))
        k = int(rng.integers(32, 1025))
        out.append((n, p, seed + 100 + i, dict(formulation=f, constraintParameter=s,
                                                tolerance=1e-6, maximumIterations=200,
                                                totalStartingPoints=k, batchSize=k,
                                                startMode=am.START_DEVICE_UNIFORM)))
    return out


def run_uneven(args):
    """Config 3 on one GPU: 256 independent problems of uneven shape.
    Three arms over the same matrices, settings and device-generated starts:
      plain   -- the plain FP32 path, one am24_solve_resident_f32 call per problem
                 (the drop-in solve a caller makes), wall clock around all calls;
      grouped -- every problem in one group (am24_group_run: one captured graph,
                 grouped launches per step, device loop), FP32, device-timed;
      mixed   -- the same group with MIXED precision (--mixed-lead FP32-accurate
                 steps, then single-pass FP16 V = B^T Z until the supports
                 settle, then FP32-accurate), device-timed.
    start-iterations are counted per start to its problem's own stop.  Accuracy:
    per problem, the best explained variance ||B x||^2 (FP64 on the device) of
    grouped and mixed against the plain path's."""
    import numpy as np
    import torch
    am = importlib.import_module("24am_b200")
    wl = am.workloads
    solver = am.Solver(0)
    probs = uneven_problems(am, wl, args.problems, SEED + 7)
    mats, sets = [], []
    t_gen = time.perf_counter()
    for (n, p, seed, kw) in probs:
        Dt = wl.low_rank_data_torch(n, p, max(1, min(n, p) // 20), min(64, p), seed)
        c2 = float(Dt.double().norm(dim=1).max())
        c1 = float(Dt.double().abs().sum(dim=1).max())
        torch.cuda.synchronize()
        M = am.Matrix(solver, None, on_device_ptr=Dt.data_ptr(), m=n, n=p, ldB=n)
        del Dt
        f = kw["formulation"]
        g = 0.1 * c2 if f in (4, 6) else (0.025 * c1 if f in (5, 7) else 0.0)
        mats.append(M)
        sets.append(dict(kw, penaltyParameter=g))
    torch.cuda.empty_cache()
    t_gen = time.perf_counter() - t_gen

    # plain FP32 path: one solve per problem
    plain_ev, plain_its, plain_steps = [], 0, []
    solver.sync()
    t0 = time.perf_counter()
    for M, kw in zip(mats, sets):
        x, f, st = M.solve(am.OptimizationSettings(**kw))
        plain_ev.append(st.explained_variance)
        plain_its += int(st.start_iterations)
        plain_steps.append(int(st.it))
    plain_s = time.perf_counter() - t0

    tune = {"seconds": 0.0}

    def grouped(precision):
        grp = am.Group(solver, capacity=len(mats))
        grp.set_autotune(not args.no_autotune)
        t_add = time.perf_counter()
        lead = args.mixed_lead if precision == am.PRECISION_MIXED else 0
        ids = [grp.add(M, am.OptimizationSettings(precision=precision, leadIterations=lead, **kw))
               for M, kw in zip(mats, sets)]
        tune["seconds"] += time.perf_counter() - t_add
        ms = grp.run()
        evs, its, low = [], 0, 0
        for pid in ids:
            _, st = grp.result(pid)
            evs.append(st.explained_variance)
            its += int(st.start_iterations)
            low += int(st.low_precision_iterations)
        grp.close()
        return ms, evs, its, low

    ms32, ev32, its32, _ = grouped(am.PRECISION_FP32)
    msmx, evmx, itsmx, lowmx = grouped(am.PRECISION_MIXED)
    pe = np.array(plain_ev)

    def ev_diffs(ev):
        """Relative explained-variance differences from the plain solves over
        the problems whose plain result is non-degenerate (finite, non-zero);
        the others must be degenerate on both sides."""
        ev = np.array(ev)
        ok = np.isfinite(pe) & (pe > 0)
        both_degenerate = int((~ok & ~(np.isfinite(ev) & (ev > 0))).sum())
        rel = np.abs(ev[ok] - pe[ok]) / pe[ok]
        rel = np.where(np.isnan(rel), np.inf, rel)
        return {"max_ev_rel_diff_vs_plain": float(rel.max(initial=0.0)),
                "median_ev_rel_diff_vs_plain": float(np.median(rel)) if rel.size else 0.0,
                "problems_within_1e-4": int((rel <= 1e-4).sum()),
                "problems_compared": int(ok.sum()),
                "degenerate_on_both_sides": both_degenerate}
    v_plain = plain_its / plain_s
    v32 = its32 / (ms32 * 1e-3)
    vmx = itsmx / (msmx * 1e-3)
    ks = [kw["totalStartingPoints"] for kw in sets]
    line = {"metric": "start-iterations/s (uneven problems, mixed precision, grouped)",
            "value": vmx, "unit": "start-it/s", "n_gpus": 1, "higher_is_better": True,
            "dtype": "bf16+f32", "data": "synthetic",
            "config": {"workload": f"{len(mats)} independent problems, each its own matrix: "
                                   "n log-uniform 100..5000 x p log-uniform 1e3..1e5, "
                                   "r = min(n,p)/20, 64 nnz/loading; formulation uniform, "
                                   "s 8..256, starts 32..1024 (device U[-1,1]), maxIter 200, "
                                   "tol 1e-6",
                       "total_starts": int(sum(ks)),
                       "mixed_lead_iterations": args.mixed_lead,
                       "matrix_elements": int(sum(n * p for n, p, _, _ in probs))},
            "plain_fp32": {"value": v_plain, "seconds": plain_s, "start_iterations": plain_its,
                           "timing": "wall clock around one am24_solve_resident_f32 per problem"},
            "grouped_fp32": dict({"value": v32, "device_ms": ms32,
                                  "start_iterations": its32}, **ev_diffs(ev32)),
            "grouped_mixed": dict({"value": vmx, "device_ms": msmx, "start_iterations": itsmx,
                                   "low_precision_step_share":
                                       lowmx / max(1, sum(plain_steps))}, **ev_diffs(evmx)),
            "speedup_mixed_vs_plain": vmx / v_plain,
            "speedup_grouped_fp32_vs_plain": v32 / v_plain,
            "speedup_mixed_vs_grouped_fp32": vmx / v32,
            "setup_seconds": t_gen,
            "group_add_seconds": tune["seconds"],
            "autotune": (not args.no_autotune,
                         "tiles per problem bucket timed once (N tile, split-K); the adds "
                         "of both grouped arms, outside the timed runs")}
    print(json.dumps(line), flush=True)
    for M in mats:
        M.close()
    solver.close()
    return 0


def corpus_csc(m, n, nnz, seed):
    """A bag-of-words-like CSC matrix: m documents x n terms, about nnz entries,
    term popularity Zipf-like (p_t ~ 1 / (t + 10)^1.1), documents uniform,
    counts-like positive values; duplicates summed.  Returns (scipy CSC,
    column means)."""
    import numpy as np
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    p = 1.0 / (np.arange(n) + 10.0) ** 1.1
    p /= p.sum()
    cols = rng.choice(n, size=nnz, p=p).astype(np.int32)
    rows = rng.integers(0, m, nnz, dtype=np.int32)
    vals = (1.0 + rng.exponential(1.0, nnz)).astype(np.float32)
    S = sp.csc_matrix((vals, (rows, cols)), shape=(m, n), dtype=np.float32)
    S.sum_duplicates()
    mu = np.asarray(S.mean(axis=0), np.float32).ravel()
    return S, mu


def run_sparse(args):
    """Sparse (CSC) input, column-centred as the reference's text-corpus runs
    are: whole solves of a fixed number of steps (tolerance 0) from device
    starts, on the sparse-resident matrix and, where its dense form fits, on
    the densified one.  start-iterations/s from the library's CUDA-event time
    of the iterations."""
    import numpy as np
    am = importlib.import_module("24am_b200")
    solver = am.Solver(0)
    cases = [("corpus 200000 x 100000, 20M nnz", 200_000, 100_000, 20_000_000, False),
             ("20000 x 50000 at 1 % density", 20_000, 50_000, 10_000_000, True)]
    out = []
    for name, m, n, nnz, dense_too in cases:
        t0 = time.perf_counter()
        S, mu = corpus_csc(m, n, nnz, SEED)
        gen_s = time.perf_counter() - t0
        row = {"case": name, "m": m, "n": n, "nnz": int(S.nnz), "generate_s": gen_s}
        for keep in ([True, False] if dense_too else [True]):
            t0 = time.perf_counter()
            M = am.Matrix.from_csc(solver, S, None, None, None, None, means=mu, keep_sparse=keep)
            solver.sync()
            up_s = time.perf_counter() - t0
            res = {"upload_s": up_s}
            for f, kw in ((0, dict(constraintParameter=32)), (3, dict(constraintParameter=32))):
                st = am.OptimizationSettings(formulation=f, tolerance=0.0, maximumIterations=20,
                                             totalStartingPoints=1024, batchSize=1024,
                                             startMode=am.START_DEVICE_UNIFORM, **kw)
                M.solve(st)  # warm-up: module loading, pool growth
                _, fval, s = M.solve(st)
                res[f"form{f}"] = {"start_it_per_s": s.start_iterations / s.total_true_computation_time,
                                   "ms_per_step": 1e3 * s.total_true_computation_time / max(1, s.it),
                                   "explained_variance": s.explained_variance}
            M.close()
            row["sparse_resident" if keep else "densified"] = res
        out.append(row)
    v = out[0]["sparse_resident"]
    vals = [v[k]["start_it_per_s"] for k in v if k.startswith("form")]
    line = {"metric": "start-iterations/s (sparse CSC input, column-centred)",
            "value": float(np.mean(vals)), "unit": "start-it/s", "n_gpus": 1,
            "higher_is_better": True, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "bag-of-words-like CSC (Zipf term popularity), column means "
                                   "subtracted implicitly; 1024 device starts; forms 0 and 3 "
                                   "(s = 32); 20 steps per solve",
                       "value_case": out[0]["case"]},
            "cases": out}
    print(json.dumps(line), flush=True)
    solver.close()
    return 0


def run_serving(args):
    """The serving layer on one GPU.  Resident matrices from the uneven-problem
    distribution (p log-uniform in [1e3, 1e5], n log-uniform in [100, 5000],
    r = min(n, p) / 20, 64 non-zeros per loading) under a 150 GB budget.
    Poisson arrivals at each rate for --seconds (at most --max-requests of
    them), then the queue drains; latency is submission to completion as the
    library measures it.  The sustained rate is the highest offered rate the
    server completes at (solves/s within 10 % of it); p99 there is the bound
    the line states."""
    import numpy as np
    import torch
    am = importlib.import_module("24am_b200")
    wl = am.workloads
    rng = np.random.default_rng(SEED)
    srv = am.Server(0, 150 << 30)
    mats, keep = [], []
    for i in range(args.matrices):
        n = int(np.exp(rng.uniform(np.log(100), np.log(5000))))
        p = int(np.exp(rng.uniform(np.log(1000), np.log(100000))))
        Dt = wl.low_rank_data_torch(n, p, max(1, min(n, p) // 20), 64, SEED + 100 + i)
        c2 = float(Dt.double().norm(dim=1).max())
        c1 = float(Dt.double().abs().sum(dim=1).max())
        torch.cuda.synchronize()
        mid = srv.add_matrix(on_device_ptr=Dt.data_ptr(), m=n, n=p, ldB=n)
        mats.append((mid, n, p, c2, c1))
        del Dt
    torch.cuda.empty_cache()
    shapes = [(m, n) for _, m, n, _, _ in mats]
    rates = [float(r) for r in args.rates.split(",")]
    per_rate, failures = [], []
    for ri, rate in enumerate(rates):
        window = min(args.seconds, args.max_requests / rate)
        reqs = config3_problems(am, int(rate * window * 2) + 50, mats, SEED + 1000 + ri)
        gaps = rng.exponential(1.0 / rate, size=len(reqs))
        tickets = []
        t0 = time.perf_counter()
        nxt = t0
        for (mid, _, st), g in zip(reqs, gaps):
            nxt += g
            if nxt - t0 > window or len(tickets) >= args.max_requests:
                break
            delay = nxt - time.perf_counter()
            if delay > 0:
                time.sleep(delay)
            try:
                tickets.append(srv.submit(mid, st))
            except am.Am24Error as e:
                failures.append(str(e))
                break
        lat, its = [], 0
        for t in tickets:
            try:
                _, s = srv.wait(t)
            except am.Am24Error as e:
                failures.append(str(e))
                continue
            lat.append(s.total_elapsed_time * 1e3)
            its += int(s.start_iterations)
        span = time.perf_counter() - t0
        lat = np.array(lat) if lat else np.array([np.nan])
        per_rate.append({"rate_req_s": rate, "requests": len(tickets),
                         "completed": int(np.isfinite(lat).sum()),
                         "arrival_window_s": window,
                         "solves_per_s": int(np.isfinite(lat).sum()) / span,
                         "p50_ms": float(np.percentile(lat, 50)),
                         "p99_ms": float(np.percentile(lat, 99)),
                         "start_it_per_s": its / span, "seconds": span})
        if failures:
            print(f"serving: {len(failures)} failed requests at {rate} req/s; first: "
                  f"{failures[0]}", file=sys.stderr, flush=True)
            break
    for r in per_rate:
        r["keeps_up"] = r["solves_per_s"] >= 0.9 * r["rate_req_s"] * min(
            1.0, r["requests"] / max(1.0, r["rate_req_s"] * r["arrival_window_s"]))
    kept = [r for r in per_rate if r["keeps_up"]]
    sustained = max(kept, key=lambda r: r["rate_req_s"]) if kept else None
    best = max(per_rate, key=lambda r: r["solves_per_s"])
    line = {"metric": "solves/s with p50/p99 latency (serving)", "value": best["solves_per_s"],
            "unit": "solves/s", "n_gpus": 1, "higher_is_better": True, "dtype": "f32",
            "data": "synthetic",
            "config": {"workload": f"Poisson requests over {len(mats)} resident matrices "
                                   "(p log-uniform 1e3..1e5, n log-uniform 100..5000), "
                                   "formulation uniform, s 8..256, starts 32..1024, maxIter 200, "
                                   "tol 1e-6, 150 GB admission budget",
                       "matrices": shapes, "arrivals_per_rate_s": args.seconds},
            "rates": per_rate,
            "sustained_rate_req_s": sustained["rate_req_s"] if sustained else None,
            "p99_bound_ms_at_sustained": sustained["p99_ms"] if sustained else None,
            "p50_ms_at_sustained": sustained["p50_ms"] if sustained else None,
            "failed_requests": len(failures),
            "first_failure": failures[0] if failures else None}
    print(json.dumps(line), flush=True)
    srv.close()
    return 1 if failures else 0


PRECISION_NOTE = ("FP32-accurate products, FP32 accumulate: both products on split FP16 "
                  "operands with power-of-two scales (h0 + h1 per operand, 22 significant "
                  "bits; Z of the L1-variance forms an exact sign), Z = B V of sparse V as an "
                  "FP32 gather")


def gemm_scheme(f):
    """Operand scheme of V = B^T Z for formulation f: on CTA pairs (more than
    128 starts) split FP16 (two MMAs per product for the L1-variance forms 1, 3,
    5, 7, whose Z is an exact sign; three for the others), or with
    AM24_GEMM_FP16=0 three BF16 MMAs for the L1-variance forms; else 3xTF32."""
    pair = STARTS > 128 and os.environ.get("AM24_GEMM_PAIR", "1") != "0"
    if pair and os.environ.get("AM24_GEMM_FP16", "1") != "0":
        return "fp16x2" if f in (1, 3, 5, 7) else "fp16x3"
    if pair and f in (1, 3, 5, 7) and os.environ.get("AM24_GEMM_BF16", "1") != "0":
        return "bf16x3"
    return "tf32x3"


def kernel_label(kind, f):
    """Bench name of a step kernel of formulation f: V = B^T Z by operand scheme
    (gemm_scheme) and epilogue (raw for the constrained forms, fused penalty
    otherwise); the select by constraint (top-s for 0, 1; L1 ball for 2, 3)."""
    skipped = kind.endswith("(skipped)")
    base = kind[:-len("(skipped)")] if skipped else kind
    if base == "gemm_BtZ":
        base = f"gemm_BtZ_{gemm_scheme(f)}_{'raw' if f <= 3 else 'pen'}"
    elif base == "select":
        base = "select_top_s" if f in (0, 1) else "select_l1_ball"
    return base + ("(skipped)" if skipped else "")


def memory_bound_rooflines(per_kind, pk, pk_kind):
    """The HBM-bound passes of the timed steps against the HBM peak, with
    algorithmic bytes per launch: the selects p*k*4 (read V = B^T Z) +
    p*k*4 (write X), as if unfused; densify p*k*4 (read V) + p*k*4 (its two
    FP16 planes); the sparse gather its B rows (every start's non-zeros times
    n samples, FP32) + n*k*4 (write Z), most rows served from L2.  The selects
    read only the candidates V = B^T Z's epilogue marked, so their rate over
    the unfused figure can pass the peak: that is the fusion's gain, not
    bandwidth."""
    out = {}
    pk_bw = pk["hbm_gbs"]
    for key, v in per_kind.items():
        if "skipped" in key:
            continue
        if key.startswith("select"):
            byts = 8.0 * P_FEATURES * STARTS
            note = "p*k*(4 read + 4 write), unfused figure"
        elif key.startswith("densify"):
            byts = 8.0 * P_FEATURES * STARTS
            note = "p*k*(4 read + 4 write)"
        else:
            continue
        avg = statistics.mean(v)
        gbs = byts / (avg * 1e-3) / 1e9
        out[key] = {"avg_launch_ms": avg, "algorithmic_bytes": byts, "achieved_gbs": gbs,
                    "peak_gbs": pk_bw, "frac": gbs / pk_bw, "bytes_note": note,
                    "traffic": profiled_traffic(key), "peak_kind": pk_kind}
    return out


def run_ours(args):
    import numpy as np
    import torch
    rank, world, local = dist_env()
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=300))
    torch.cuda.set_device(local)
    am = importlib.import_module("24am_b200")
    wl = am.workloads
    solver = am.Solver(local)
    stream = torch.cuda.ExternalStream(solver.stream())

    Dt = wl.low_rank_data_torch(N_SAMPLES, P_FEATURES, RANK, NNZ_V, SEED)  # (p, n): B col-major
    col2 = float(Dt.double().norm(dim=1).max())
    col1 = float(Dt.double().abs().sum(dim=1).max())
    gam = wl.penalty_gammas(col2, col1, GAMMA_C)
    torch.cuda.synchronize()
    M = am.Matrix(solver, None, on_device_ptr=Dt.data_ptr(), m=N_SAMPLES, n=P_FEATURES,
                  ldB=N_SAMPLES)
    forms = [int(x) for x in args.formulations.split(",")]
    batches, starts = [], []
    for f in forms:
        V = wl.uniform_starts_torch(P_FEATURES, STARTS, seed=1000 + SEED + 17 * rank + f)
        torch.cuda.synchronize()
        st = am.OptimizationSettings(formulation=f, constraintParameter=S_CONS,
                                     penaltyParameter=gam.get(f, 0.0), tolerance=E2E_TOL,
                                     maximumIterations=E2E_MAX_IT, totalStartingPoints=STARTS,
                                     batchSize=STARTS)
        b = M.batch(st, STARTS)
        b.load(device_ptr=V.data_ptr())
        batches.append(b)
        starts.append(V)
    launches_per_step = sum(b.launches_per_step() for b in batches)

    def step(it):
        for b in batches:
            b.iterate(it, 1, sync=False)

    def barrier():
        if world > 1:
            torch.distributed.barrier()

    for i in range(args.warmup):
        step(i)
    solver.sync()
    barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local, args.clock_ms) as clk:
        e0.record(stream)
        for i in range(args.steps):
            step(args.warmup + i)
        e1.record(stream)
        solver.sync()
    torch.cuda.synchronize()
    barrier()
    ms = e0.elapsed_time(e1)
    t = torch.tensor([ms], device="cuda", dtype=torch.float64)
    if world > 1:
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    ms_max = float(t.item())
    its_per_step = len(forms) * STARTS
    value = its_per_step * args.steps * world / (ms_max * 1e-3)

    # per-kernel CUDA events inside the same kind of steps
    per_kind, per_form = {}, {}
    for i in range(max(1, min(args.steps, 5))):
        for f, b in zip(forms, batches):
            for kind, kms in b.step_timed(args.warmup + args.steps + i):
                key = kernel_label(kind, f)
                per_kind.setdefault(key, []).append(kms)
                pf = per_form.setdefault(f, {})
                pf[key] = pf.get(key, 0.0) + kms
    n_timed = max(1, min(args.steps, 5))
    formulation_ms = {str(f): {"step_ms": sum(d.values()) / n_timed,
                               "kernels": {k: v / n_timed for k, v in sorted(d.items())
                                           if "skipped" not in k}}
                      for f, d in per_form.items()}
    totals = {k: sum(v) for k, v in per_kind.items()}
    roof_kinds = {k: t for k, t in totals.items() if k.startswith(("gemm", "select"))
                  and "skipped" not in k}
    dom = max(roof_kinds, key=roof_kinds.get)
    pk, pk_kind = peaks()
    avg_ms = statistics.mean(per_kind[dom])
    if dom.startswith("gemm"):
        # FP32-equivalent rate: 2*n*p*k FLOPs per launch against the tensor
        # rate of the scheme's passes (three TF32 MMAs at half the 16-bit
        # rate, or three or two BF16 / FP16 MMAs, per FP32 product)
        passes = {"fp16x2": 2.0, "fp16x3": 3.0, "bf16x3": 3.0, "tf32x3": 6.0}
        scheme = next(s for s in passes if s in dom)
        div = passes[scheme]
        # the kernel's time comes from its own CUDA events around one launch
        # (am24_batch_step_timed), i.e. the kernel timed alone: the burst peak
        peak = pk["bf16_tflops"] / div
        flops = 2.0 * N_SAMPLES * P_FEATURES * STARTS
        achieved = flops / (avg_ms * 1e-3) / 1e12
        roof = {"bound": "tensor", "achieved": achieved, "peak": peak, "unit": "TFLOP/s",
                "frac": achieved / peak, "traffic": profiled_traffic(dom),
                "kernel": dom, "avg_launch_ms": avg_ms,
                "frac_of_sustained": achieved / (pk["bf16_tflops_sustained"] / div),
                "peak_note": f"{pk_kind} bf16 burst {pk['bf16_tflops']} TF/s"
                             + {"fp16x2": " /2 (two FP16 MMAs per FP32 product)",
                                "fp16x3": " /3 (three FP16 MMAs per FP32 product)",
                                "bf16x3": " /3 (three BF16 MMAs per FP32 product)",
                                "tf32x3": " /2 (TF32 rate) /3 (three TF32 MMAs per FP32 "
                                          "product)"}[scheme]
                             + "; achieved counts 2*n*p*k dense FLOPs per launch"}
    else:
        byts = 4.0 * P_FEATURES * STARTS * 3
        achieved = byts / (avg_ms * 1e-3) / 1e9
        roof = {"bound": "hbm", "achieved": achieved, "peak": pk["hbm_gbs"], "unit": "GB/s",
                "frac": achieved / pk["hbm_gbs"], "traffic": profiled_traffic(dom),
                "kernel": dom, "avg_launch_ms": avg_ms}
    breakdown = {k: {"launches": len(v), "avg_ms": statistics.mean(v),
                     "share": totals[k] / sum(totals.values())} for k, v in per_kind.items()}
    memory_bound = memory_bound_rooflines(per_kind, pk, pk_kind)

    # e2e through the one-call public API with pinned host buffers
    e2e = None
    if not args.no_e2e:
        Bh = Dt.cpu().pin_memory()  # (p, n) contiguous == n x p column-major
        x = torch.zeros(P_FEATURES, dtype=torch.float32).pin_memory()
        t_e2e, its_e2e, h2d, d2h = 0.0, 0, 0, 0
        # untimed warm-up passes first (module loading, memory pool growth),
        # as for the device-timed steps
        for rep in range(max(0, args.e2e_warmup) + max(1, args.e2e_steps)):
            timed = rep >= max(0, args.e2e_warmup)
            for fi, f in enumerate(forms):
                Vh = starts[fi].cpu().pin_memory()
                st = am.OptimizationSettings(formulation=f, constraintParameter=S_CONS,
                                             penaltyParameter=gam.get(f, 0.0), tolerance=E2E_TOL,
                                             maximumIterations=E2E_MAX_IT,
                                             totalStartingPoints=STARTS, batchSize=STARTS,
                                             startMode=am.START_INJECTED)
                s_c = st.to_c()
                stc = am.am24_statistics()
                fv = C.c_float()
                barrier()
                t0 = time.perf_counter()
                am.check(am.lib().am24_solve_dense_f32(
                    solver.h, C.c_void_p(Bh.data_ptr()), N_SAMPLES, C.c_void_p(x.data_ptr()),
                    N_SAMPLES, P_FEATURES, C.byref(s_c), C.byref(stc),
                    C.c_void_p(Vh.data_ptr()), C.byref(fv)))
                if not timed:
                    continue
                t_e2e += time.perf_counter() - t0
                its_e2e += int(stc.start_iterations)
                h2d += Bh.numel() * 4 + Vh.numel() * 4
                d2h += x.numel() * 4
        tt = torch.tensor([t_e2e], device="cuda", dtype=torch.float64)
        if world > 1:
            torch.distributed.all_reduce(tt, op=torch.distributed.ReduceOp.MAX)
        steps_e2e = max(1, args.e2e_steps)
        e2e = {"value": its_e2e * world / float(tt.item()), "unit": "start-it/s",
               "h2d_bytes_per_step": h2d // steps_e2e, "d2h_bytes_per_step": d2h // steps_e2e,
               "solves_per_step": len(forms), "start_iterations": its_e2e,
               "warmup": max(0, args.e2e_warmup),
               "note": "am24_solve_dense_f32 per formulation, maxIter 200, tol 1e-6, "
                       "pinned host B and starts, wall clock around each call, after "
                       "untimed warm-up passes over the same solves"}

    cpu = None
    if world == 1 and rank == 0 and not args.no_cpu:
        Bnp = Dt.cpu().numpy().T  # n x p view, column-major
        import numpy as np
        Bnp = np.asfortranarray(Bnp)
        v, cores, kind, its, secs, starts, code = cpu_sample(Bnp)
        cpu = {"value": v, "unit": "start-it/s", "cores": cores, "kind": kind,
               "sample": f"8 formulations x {CPU_SAMPLE_ITERS} iterations x "
                         f"{starts} starts on the full matrix ({its} start-iterations, "
                         f"{secs:.1f} s compute, {code})"}
        if not args.no_oracle_check:
            t0 = time.perf_counter()
            cpu["fp64_oracle_check"] = {
                "per_formulation": fp64_oracle_check(am, M, Bnp, gam, 256, CPU_SAMPLE_ITERS),
                "how": f"256 reference starts (CTA-pair tiles, split-FP16 products, as the "
                       f"timed steps run) x {CPU_SAMPLE_ITERS} steps on the device against the "
                       "FP64 oracle from the same starts; starts with an ill-conditioned "
                       "decision (FP32-size ties) set aside",
                "seconds": time.perf_counter() - t0}

    if rank == 0:
        line = {"metric": "start-iterations/s", "value": value, "unit": "start-it/s",
                "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
                "ms_per_step": ms_max / args.steps, "higher_is_better": True, "scaling": "weak",
                "vs_baseline": None, "dtype": "f32", "data": "synthetic",
                "config": bench_config(world, forms),
                "roofline": roof, "memory_bound": memory_bound, "kernels": breakdown,
                "formulation_ms": formulation_ms,
                "cpu_baseline": cpu, "e2e": e2e,
                "gpu_launches": launches_per_step * args.steps,
                "clocks": clk.summary()}
        print(json.dumps(line), flush=True)
    for b in batches:
        b.close()
    M.close()
    solver.close()
    if world > 1:
        torch.distributed.destroy_process_group()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--clock-ms", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=1)
    ap.add_argument("--e2e-warmup", type=int, default=1)
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-oracle-check", action="store_true",
                    help="skip the per-start FP64 oracle check after the CPU baseline")
    ap.add_argument("--size", default="config1", choices=sorted(SIZES))
    ap.add_argument("--formulations", default=None,
                    help="subset for profiling runs; the headline uses all 8 "
                         "(config2: 0 and 7, its two forms)")
    ap.add_argument("--mode", default="step",
                    choices=["step", "solve", "serve", "uneven", "sparse"],
                    help="step: the AM-step throughput line; solve: whole solves to tol, "
                         "FP32 and MIXED precision from the same starts; serve: Poisson "
                         "requests to the serving layer (p50/p99 latency); uneven: 256 "
                         "problems of uneven shapes submitted at once; sparse: CSC input kept "
                         "compressed on the device against its densified form")
    ap.add_argument("--rates", default="10,30,100,300,1000,2000",
                    help="serve: request rates (req/s)")
    ap.add_argument("--max-requests", type=int, default=400,
                    help="serve: arrivals per rate at most")
    ap.add_argument("--seconds", type=float, default=5.0, help="serve: arrivals per rate")
    ap.add_argument("--matrices", type=int, default=32, help="serve: resident matrices")
    ap.add_argument("--problems", type=int, default=256, help="uneven: problems")
    ap.add_argument("--no-autotune", action="store_true", help="uneven: cost-model tiles")
    ap.add_argument("--mixed-lead", type=int, default=20,
                    help="solve / uneven: FP32-accurate iterations before MIXED's single-pass "
                         "phase (0: single-pass from the first iteration)")
    args = ap.parse_args()
    global N_SAMPLES, P_FEATURES, RANK, NNZ_V, STARTS, S_CONS, GAMMA_C
    N_SAMPLES, P_FEATURES, RANK, NNZ_V, STARTS = SIZES[args.size]
    S_CONS = SIZE_S[args.size]
    GAMMA_C = SIZE_GAMMA[args.size]
    if args.formulations is None:
        args.formulations = "0,7" if args.size == "config2" else "0,1,2,3,4,5,6,7"
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        return run_reference_arm(args)
    if args.mode == "solve":
        return run_solves(args)
    if args.mode == "uneven":
        return run_uneven(args)
    if args.mode == "serve":
        return run_serving(args)
    if args.mode == "sparse":
        return run_sparse(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
