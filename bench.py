"""Benchmark: seconds per pressure solve to a 1e-10 relative residual on a
256^3 jittered, permuted hex mesh (16.8M cells, 50.1M interior faces):
the learned + mixed-precision solve against plain FP64 PCG, plus the HBM
rooflines of the kernels that dominate it.

One step = one full solve of the pressure-correction Poisson system
(jitter +-15%, cells randomly permuted (seed 0) then renumbered by the
framework (reverse Cuthill-McKee), coefficients area/l_pn, all-Neumann
boundaries, cell 1 pinned, rhs uniform[-1,1] with its mean removed,
phi0 = 0) with the spray-simulation stopping rule |r|_1/|r0|_1 < 1e-10.

  python bench.py [--gpus N --steps K --warmup W] [--impl reference]
                  [--size 256] [--method learned|mg_jacobi|mixed|plain]
                  [--no-configs] [--no-cpu] [--no-tune]

Methods (all through the library's C-ABI, same context, same system):
  learned   -- flexible CG, FP32 inner iteration with FP64 reliable
               updates, preconditioned by one V-cycle of the aggregation
               hierarchy whose finest-level smoother is the network's
               operator (solv_gpu_fcg); `value`
  mg_jacobi -- the same V-cycle with damped-Jacobi smoothing (no network)
  one_level -- the network's operator alone as the preconditioner
  mixed     -- Jacobi PCG, FP32 inner iteration with FP64 reliable updates
  plain     -- Jacobi PCG in FP64 (solv_gpu_cg, the reference algorithm)
Each is timed with CUDA events on the solver's stream (inputs resident in
HBM; every array is larger than the 126 MB L2, so no flush is needed); the
measured method is then timed end to end through the host C-ABI with
pinned host buffers (`e2e`).  The hierarchy is built once per mesh (host
aggregation) by the first solve, outside the timed region, like the matrix
structure itself: `first_call_s` reports that first solve.

The other configurations are timed after the headline and reported as
extra keys (`configs`): the 32^3 plain PCG of the reference's own scale,
BiCGSTAB + DILU on the 128^3 momentum system in FP64 and with FP32 inner
iterations (in RCM order and in the multicolour order), and the batched
solves (u, v, w on one 96^3 mesh; 64 uneven meshes of 8k-500k cells).

The reference arm (--impl reference) and `cpu_baseline` time the CPU
oracle -- the line-faithful C restatement of the Fortran solver, single
core like the reference -- on a bounded sample of iterations of the same
system, and extrapolate to the full solve with the ORACLE's own iteration
count (a full 256^3 oracle solve, tests/golden/oracle_pcg_256.json; smaller
sizes are solved in full).  The extrapolation is checked against full
oracle solves at 32^3 and 64^3, printed in the line.
Multi-GPU: the path does not shard (replicas only): each rank solves its
own system; timing is the max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

PEAK_FALLBACK_GBS = 6650.0
METRIC = "s/solve to 1e-10 rel resid (learned+mixed vs plain FP64 PCG); SpMV HBM GB/s"
STEP_SAMPLE_S = 8.0   # CPU seconds of oracle iterations per reference-arm step


def _env_int(k, d):
    try:
        return int(os.environ.get(k, d))
    except ValueError:
        return d


def max_over_ranks(x, dist=None, device=None):
    """The largest of every rank's x: a job of replicas takes as long as its
    slowest rank.  Every rank must call it, in the same order."""
    if dist is None:
        return float(x)
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def host_cpu():
    """The host the CPU baseline ran on: model name and hardware threads."""
    model = None
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    model = line.split(":", 1)[1].strip()
                    break
    except OSError:
        pass
    return {"cpu_model": model, "host_threads": os.cpu_count()}


def _peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return PEAK_FALLBACK_GBS, "fallback"


def build_system(size: int, seed: int = 0):
    from programs_b200.mesh import Mesh, poisson_rhs
    m = Mesh.hex(size, jitter=0.15, seed=seed, permute=True)
    m.renumber(Mesh.RCM)
    A = m.pressure(pin=1)
    b = poisson_rhs(A.n_cell, seed + 1)
    del m
    return A, b


def n_interior(A):
    return int((A.inb > 0).sum())


def spmv_bytes(A, fp=8, k=1):
    """Algorithmic bytes of one matrix product: F*(8+fp*k) + 3*fp*N
    (index pair + k coefficients per interior face; diag, x, y per cell)."""
    return n_interior(A) * (8 + fp * k) + 3 * fp * A.n_cell


# Algorithmic bytes per launch of the kernels kernel_time() can time (F
# interior faces, N cells; FP32 unless noted): every face's index pair and
# coefficient once, and each per-cell vector once.
def kernel_bytes(A):
    F, N = n_interior(A), A.n_cell
    return {
        "spmv_fp64": F * 16 + 24 * N,            # y = A x (FP64)
        "spmv_fp32": F * 12 + 12 * N,            # y = A x (row sum, x, y)
        "net_apply": F * 12 + 12 * N,            # z = K r (q, r, z; a weight per face)
        "mg_resid": F * 12 + 16 * N,             # t = b - A x (row sum, b, x, t)
        "net_smooth": F * 12 + 12 * N,           # x = w K b
        "fcg_spmv": F * 12 + 16 * N,             # q = A p, p.q, p.r (row sum, p, r, q)
        "cg_spmv_fp64": F * 16 + 32 * N,         # q = A p, p.q (diag, p, q) FP64
        "dilu_apply_fp64": 2 * F * 16 + 80 * N,  # both recurrences: sweep coefficients,
                                                 # c, c_r, r in, t out/in, z out
    }


KERNEL_WHICH = {"spmv_fp64": 0, "spmv_fp32": 1, "net_apply": 2, "mg_resid": 4, "net_smooth": 5,
                "fcg_spmv": 6, "cg_spmv_fp64": 7, "dilu_apply_fp64": 8}


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.out = ""

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except (OSError, FileNotFoundError):
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.out, _ = self.proc.communicate(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
                self.out, _ = self.proc.communicate()

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in (self.out or "").splitlines():
            f = [x.strip() for x in line.split(",")]
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
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def _traffic_from_profile(name):
    """DRAM bytes per launch from a committed ncu summary, if present."""
    p = os.path.join(ROOT, "profiles", name)
    if not os.path.exists(p):
        return None
    for line in open(p):
        if line.startswith("dram_bytes_per_launch:"):
            try:
                return float(line.split(":", 1)[1].split()[0])
            except ValueError:
                return None
    return None


# ---- the CPU oracle: reference arm and cpu_baseline --------------------------------
def oracle_full_solve(size):
    """The oracle's own full solve of the size^3 system, where one has been
    recorded (tests/golden/oracle_pcg_<size>.json): iterations and seconds."""
    p = os.path.join(ROOT, "tests", "golden", f"oracle_pcg_{size}.json")
    if not os.path.exists(p):
        return None
    with open(p) as f:
        d = json.load(f)
    return {"iterations": int(d["iterations"]), "solve_s": float(d["solve_s"]),
            "sample_idx": d["sample_idx"], "sample_x": d["sample_x"]}


def _oracle_iteration_s(o, b, n):
    t = time.perf_counter()
    o.solv_cg(0, 1e-10, n, np.zeros((o.N, 1)), b.reshape(-1, 1))
    return (time.perf_counter() - t) / n


def oracle_cost(o, b, n_long, n_short=1):
    """(seconds per PCG iteration, fixed seconds per call) of the oracle on
    this system, from one call of n_short and one of n_long iterations: the
    difference removes what every call pays once (the initial residual, the
    preconditioner, the work arrays' first touch)."""
    t1 = _oracle_iteration_s(o, b, n_short) * n_short
    t2 = _oracle_iteration_s(o, b, n_long) * n_long
    per = max(t2 - t1, 0.0) / max(n_long - n_short, 1)
    return per, max(t1 - n_short * per, 0.0)


def oracle_iterations(A, b, size):
    """The oracle's iteration count for this system: recorded for the large
    sizes, solved in full here otherwise."""
    full = oracle_full_solve(size)
    if full is not None:
        return full["iterations"], "recorded full oracle solve (tests/golden)"
    from oracle.oracle import Oracle
    r = Oracle.from_matrix(A).solv_cg(0, 1e-10, 100000, np.zeros((A.n_cell, 1)),
                                      b.reshape(-1, 1))
    return int(r[3][0]), "full oracle solve, this run"


def extrapolation_check(sizes=(32, 64), sample=20):
    """Full oracle solves against the extrapolation the CPU baseline uses
    (fixed cost + seconds per iteration x iterations), at sizes the oracle
    finishes in seconds."""
    from oracle.oracle import Oracle
    out = {}
    for n in sizes:
        A, b = build_system(n)
        o = Oracle.from_matrix(A)
        per, fixed = oracle_cost(o, b, min(sample, 50))
        t = time.perf_counter()
        r = o.solv_cg(0, 1e-10, 100000, np.zeros((A.n_cell, 1)), b.reshape(-1, 1))
        full = time.perf_counter() - t
        it = int(r[3][0])
        est = fixed + per * it
        out[f"{n}^3"] = {"iterations": it, "full_solve_s": full,
                         "extrapolated_s": est, "extrapolated_over_full": est / full}
    return out


def cpu_oracle_sample(A, b, budget_s, repeats=1):
    """The oracle's cost on this system (single core: the reference is
    serial): `repeats` samples of about budget_s seconds, each a short and a
    long call; returns ([seconds per iteration], [fixed seconds per call],
    iterations of the long call)."""
    from oracle.oracle import Oracle
    o = Oracle.from_matrix(A)
    per0, _ = oracle_cost(o, b, 3)
    s = max(4, min(400, int(budget_s / max(per0, 1e-6))))
    out = [oracle_cost(o, b, s) for _ in range(repeats)]
    return [p for p, _ in out], [f for _, f in out], s


def _config(args, A):
    return {"workload": f"pressure Poisson {args.size}^3 jittered hex, solve to 1e-10 L1-relative",
            "n_cell": A.n_cell, "n_face_interior": n_interior(A),
            "method": args.method, "baseline_method": "plain FP64 Jacobi PCG",
            "ordering": "RCM", "l2": "inputs larger than L2 (no flush needed)",
            "parallelism": "replicas"}


def run_reference(args, rank):
    if rank != 0:
        return
    A, b = build_system(args.size, seed=0)
    iters, iters_src = oracle_iterations(A, b, args.size)
    from oracle.oracle import Oracle
    o = Oracle.from_matrix(A)
    per0, _ = oracle_cost(o, b, 3)
    sample = max(4, min(400, int(STEP_SAMPLE_S / max(per0, 1e-6))))
    for _ in range(args.warmup):
        _oracle_iteration_s(o, b, 1)
    per, fixed, step_s = [], [], []
    for _ in range(args.steps):
        t = time.perf_counter()
        p_, f_ = oracle_cost(o, b, sample)
        per.append(p_)
        fixed.append(f_)
        step_s.append(time.perf_counter() - t)
    v = statistics.mean(fixed) + statistics.mean(per) * iters
    check = extrapolation_check()
    desc = (f"EXTRAPOLATED: each step times one 1-iteration and one {sample}-iteration oracle "
            f"PCG call on the {args.size}^3 system (single core; the reference is serial); "
            f"value = the fixed cost of a call + mean seconds per iteration (their difference) "
            f"x the oracle's own {iters}-iteration full solve ({iters_src}); ms_per_step is the "
            f"time each step actually took")
    print(json.dumps({
        "impl": "reference", "metric": METRIC, "value": v, "unit": "s/solve",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": statistics.mean(step_s) * 1e3, "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": _config(args, A),
        "oracle_iterations": iters, "oracle_iterations_source": iters_src,
        "extrapolation_check": check,
        "cpu_baseline": {"value": v, "unit": "s/solve", "cores": 1, "kind": "port",
                         "sample": desc, **host_cpu()},
        "e2e": {"value": v, "unit": "s/solve", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }))


# The solve methods, as options of one library context.
METHODS = {
    "learned": {"solver": "fcg", "precision": 1, "mg_levels": 12, "smoother": 1},
    "mg_jacobi": {"solver": "fcg", "precision": 1, "mg_levels": 12, "smoother": 0},
    "one_level": {"solver": "fcg", "precision": 1, "mg_levels": 0, "smoother": 1},
    "mixed": {"solver": "cg", "precision": 1, "mg_levels": 12, "smoother": 1},
    "plain": {"solver": "cg", "precision": 0, "mg_levels": 12, "smoother": 1},
}


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def time_configs(s, torch, dev):
    """The other benchmark configurations, each timed with the library's own
    CUDA events (stats.solve_ms, the device time of the solve), best of the
    repeats after a first (warm-up) solve."""
    from programs_b200.cases import batch_meshes, make_system
    from programs_b200.mesh import Mesh, poisson_rhs, uniform
    from programs_b200.solver import OPT_PRECISION

    def timed_solve(kind, imat, V, b_cols, repeat=3, precision=0):
        s.set_option(OPT_PRECISION, precision)
        N = b_cols.shape[0]
        bd = torch.from_numpy(np.asfortranarray(b_cols).ravel(order="F")).to(dev)
        phi = torch.zeros(N * V, dtype=torch.float64, device=dev)
        res0 = torch.empty_like(bd)
        best, st = None, None
        for k in range(repeat + 1):
            phi.zero_()
            res0.copy_(bd)
            torch.cuda.synchronize()
            fn = s.solv_cg_dev if kind == "cg" else s.solv_bicg_dev
            _, st = fn(imat, 1e-10, 100000, V, phi.data_ptr(), res0.data_ptr())
            if k > 0:
                best = st["solve_ms"] if best is None else min(best, st["solve_ms"])
        s.set_option(OPT_PRECISION, 0)
        it = int(max(st["iters"][:V]))
        return {"s_per_solve": best / 1e3, "iterations": it, "ms_per_iteration": best / max(it, 1),
                "status": st["status"], "refinements": st["refinements"]}

    out = {}
    # C1: 32^3 as configured (permuted order as given), FP64 Jacobi PCG
    m = Mesh.hex(32, jitter=0.15, seed=0, permute=True)
    A = m.pressure(pin=1)
    s.matrix_set(A)
    b = poisson_rhs(A.n_cell, 1).reshape(-1, 1)
    out["pressure_32_plain_pcg"] = timed_solve("cg", 0, 1, b)
    # C2: 128^3 momentum, BiCGSTAB + DILU, FP64 and FP32 inner, in RCM order
    # (the recurrences 382 levels deep) and in the multicolour order (2
    # levels; a different factorisation, so other iteration counts)
    for order in ("rcm", "color"):
        A, b = make_system(128, "momentum", renumber=order)
        s.matrix_set(A)
        c2 = {"sweep_levels": s.levels}
        for name, prec in (("fp64", 0), ("fp32_inner", 1)):
            c2[name] = timed_solve("bicg", 2, 1, b.reshape(-1, 1), precision=prec)
        out[f"momentum_128_bicgstab_dilu_{order}"] = c2
    # C3a: u, v, w on one 96^3 mesh (shared matrix), BiCGSTAB + DILU, FP32
    # inner, in both cell orders
    for order in ("rcm", "color"):
        A, b = make_system(96, "momentum", renumber=order)
        s.matrix_set(A)
        B = np.stack([b, uniform(11, A.n_cell), uniform(12, A.n_cell)], axis=1)
        out[f"momentum_96_uvw_bicgstab_dilu_fp32_inner_{order}"] = timed_solve(
            "bicg", 2, 3, B, precision=1)
    # C1 again under PERSISTENT 1 (the whole loop in one launch: here the resident PCG)
    from programs_b200.solver import OPT_PERSISTENT
    m = Mesh.hex(32, jitter=0.15, seed=0, permute=True)
    A = m.pressure(pin=1)
    s.matrix_set(A)
    s.set_option(OPT_PERSISTENT, 1)
    out["pressure_32_plain_pcg_persistent"] = timed_solve("cg", 0, 1,
                                                          poisson_rhs(A.n_cell, 1).reshape(-1, 1))
    s.set_option(OPT_PERSISTENT, 0)
    # C3b: 64 uneven pressure meshes (8k-500k cells, seed 1) in one batch, FP32 inner
    mats, rhs = batch_meshes(64, 8000, 500000, seed=1)
    cp = s.matrix_set_batch(mats)
    bb = torch.from_numpy(np.concatenate(rhs)).to(dev)
    phi = torch.zeros_like(bb)
    res0 = torch.empty_like(bb)
    s.set_option(OPT_PRECISION, 1)
    best = None
    for k in range(3):
        phi.zero_()
        res0.copy_(bb)
        torch.cuda.synchronize()
        st = s.solv_batch_dev("cg", 0, 1e-10, 100000, 1, phi.data_ptr(), res0.data_ptr())
        if k > 0:
            best = st["solve_ms"] if best is None else min(best, st["solve_ms"])
    s.set_option(OPT_PRECISION, 0)
    out["pressure_batch_64_uneven_fp32_inner"] = {
        "s_per_batch": best / 1e3, "n_sys": 64, "n_cell": int(cp[-1]),
        "iters_max": int(st["iters_all"].max()), "iters_min": int(st["iters_all"].min()),
        "status": st["status"]}
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--size", type=int, default=256)
    ap.add_argument("--method", default="learned", choices=["learned", "mg_jacobi", "mixed", "plain"])
    ap.add_argument("--weights", default=None)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-tune", action="store_true")
    ap.add_argument("--no-configs", action="store_true")
    args = ap.parse_args()

    rank = _env_int("RANK", 0)
    world = _env_int("WORLD_SIZE", 1)
    local = _env_int("LOCAL_RANK", 0)
    if args.impl == "reference":
        run_reference(args, rank)
        return

    import torch
    from programs_b200.learn import DEFAULT_WEIGHTS, load_params
    from programs_b200.solver import (GpuSolver, OPT_MG_LEVELS, OPT_MG_SMOOTHER, OPT_PRECISION)
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))

    t0 = time.perf_counter()
    A, b = build_system(args.size, seed=rank)
    N = A.n_cell
    s = GpuSolver(local)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    s.matrix_set(A)
    setup_s = time.perf_counter() - t0
    s.gnn_set_params(load_params(args.weights or DEFAULT_WEIGHTS))
    dev = torch.device("cuda", local)
    b_dev = torch.from_numpy(b).to(dev).reshape(N, 1)
    phi = torch.zeros(N, 1, dtype=torch.float64, device=dev)
    res0 = torch.empty(N, 1, dtype=torch.float64, device=dev)

    def configure(method):
        m = METHODS[method]
        s.set_option(OPT_PRECISION, m["precision"])
        s.set_option(OPT_MG_LEVELS, m["mg_levels"])
        s.set_option(OPT_MG_SMOOTHER, m["smoother"])

    tune = None
    if not args.no_tune:  # the measured method's own launch shapes and vector width
        configure(args.method)
        tune = s.autotune(METHODS[args.method]["solver"], 0, 1)
    torch.cuda.synchronize()

    def solve(method, reduc=1e-10):
        configure(method)
        with torch.cuda.stream(stream):
            phi.zero_()
            res0.copy_(b_dev)
        if METHODS[method]["solver"] == "fcg":
            return s.solv_fcg_dev(reduc, 100000, phi.data_ptr(), res0.data_ptr())
        return s.solv_cg_dev(0, reduc, 100000, 1, phi.data_ptr(), res0.data_ptr())

    def first_call(method):
        torch.cuda.synchronize()
        t = time.perf_counter()
        solve(method)
        torch.cuda.synchronize()
        return time.perf_counter() - t

    def timed(method, steps, warmup, clocks=False):
        for _ in range(max(warmup, 1)):
            rn, st = solve(method)
        launches = 0
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        clk = ClockSampler(local) if clocks else None
        if clk:
            clk.__enter__()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(steps):
            rn, st = solve(method)
            launches += st["kernel_launches"] + 2
        e1.record(stream)
        torch.cuda.synchronize()
        if clk:
            clk.__exit__()
        ms = max_over_ranks(e0.elapsed_time(e1), dist, dev)
        return ms / steps, st, launches, (clk.summary() if clk else None)

    def solution():
        return phi.double().cpu().numpy().reshape(-1).copy()

    first_s = first_call(args.method)  # builds the hierarchy (once per mesh) for multigrid
    ms_step, st, launches, clocks = timed(args.method, args.steps, args.warmup, clocks=True)
    x = solution()
    S = A.to_scipy()
    true_rel = float(np.abs(b - S @ x).sum() / np.abs(b).sum())
    extra = {}
    if args.method == "learned":
        for m, k in (("mg_jacobi", 3), ("one_level", 2)):
            ms_m, st_m, _, _ = timed(m, k, 1)
            extra[m] = {"s_per_solve": ms_m / 1e3, "iterations": st_m["iters"][0]}
    ms_plain, st_plain, _, _ = (timed("plain", 2, 1) if args.method != "plain"
                                else (ms_step, st, 0, None))
    x_plain = solution()
    ms_mixed, st_mixed, _, _ = (timed("mixed", 2, 1) if args.method != "mixed"
                                else (ms_step, st, 0, None))
    # Solution agreement.  Two solves stopped at 1e-10 each carry about
    # cond(A) x 1e-10 of error; the plain FP64 solve run to 1e-12 stands in
    # for the exact solution, and the full-size oracle solve (FP64, the
    # reference's arithmetic, 1e-10) is compared at its recorded cells.
    solve("plain", 1e-12)
    x_exact = solution()
    solve(args.method, 1e-12)
    x_t = solution()
    agreement = {
        "method_vs_plain_fp64_both_at_1e-10": _rel(x, x_plain),
        "method_at_1e-10_vs_plain_fp64_at_1e-12": _rel(x, x_exact),
        "plain_fp64_at_1e-10_vs_plain_fp64_at_1e-12": _rel(x_plain, x_exact),
        "method_vs_plain_fp64_both_at_1e-12": _rel(x_t, x_exact),
    }
    full = oracle_full_solve(args.size)
    if full is not None and rank == 0:
        idx = np.asarray(full["sample_idx"])
        xo = np.asarray(full["sample_x"])
        agreement["method_at_1e-10_vs_oracle_at_1e-10_sampled"] = _rel(x[idx], xo)
        agreement["plain_fp64_at_1e-10_vs_oracle_at_1e-10_sampled"] = _rel(x_plain[idx], xo)
        agreement["oracle_at_1e-10_vs_plain_fp64_at_1e-12_sampled"] = _rel(xo, x_exact[idx])
        agreement["oracle_sample_cells"] = int(idx.size)
    del S

    # e2e: the measured method through the host C-ABI, pinned host buffers,
    # both copies inside the timed region
    phi_h = torch.zeros(N, 1, dtype=torch.float64).pin_memory().numpy()
    res_h = torch.zeros(N, 1, dtype=torch.float64).pin_memory().numpy()
    configure(args.method)
    e2e = []
    for k in range(args.steps + 1):
        phi_h[:] = 0.0
        res_h[:, 0] = b
        rn_h = np.zeros(1)
        torch.cuda.synchronize()
        t = time.perf_counter()
        if METHODS[args.method]["solver"] == "fcg":
            s.solv_fcg(1e-10, 100000, phi_h, res_h, rn_h)
        else:
            s.solv_cg(0, 1e-10, 100000, phi_h, res_h, rn_h)
        dt = time.perf_counter() - t
        if k > 0:
            e2e.append(dt)
    e2e_s = max_over_ranks(statistics.mean(e2e), dist, dev)

    # rooflines: kernels of the solves timed live on the solver's stream
    peak, peak_kind = _peaks()
    configure(args.method)
    alg = kernel_bytes(A)
    kt = {k: s.kernel_time(w, 20) for k, w in KERNEL_WHICH.items()}
    gbs = {k: alg[k] / (kt[k] * 1e-3) / 1e9 for k in kt}
    vcycle_ms = None
    if METHODS[args.method]["solver"] == "fcg":
        vcycle_ms = s.kernel_time(3, 10)
    # the dominant kernel of the measured method: the V-cycle's level-0
    # residual for the multigrid solves, the FP64 CG product for plain PCG
    dominant = {"learned": "mg_resid", "mg_jacobi": "fcg_spmv", "mixed": "spmv_fp32",
                "plain": "cg_spmv_fp64"}[args.method]
    traffic = _traffic_from_profile(f"{dominant}_pressure_{args.size}.txt")

    configs = None
    if not args.no_configs:
        configs = time_configs(s, torch, dev)

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        iters_o, src = oracle_iterations(A, b, args.size)
        per, fixed, sample = cpu_oracle_sample(A, b, 5.0, repeats=3)
        cpu = {"value": statistics.median(fixed) + statistics.median(per) * iters_o,
               "unit": "s/solve", "cores": 1, "kind": "port",
               "sample": f"EXTRAPOLATED: 3 samples of a 1- and a {sample}-iteration oracle PCG "
                         f"call on this system (single core); the fixed cost of a call + the "
                         f"median seconds per iteration (their difference) x the oracle's own "
                         f"{iters_o}-iteration full solve ({src})",
               **host_cpu()}

    if rank == 0:
        line = {
            "metric": METRIC, "value": ms_step / 1e3 / world, "unit": "s/solve", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step,
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64 (outer) / f32 (inner) / bf16 (network)" if args.method != "plain"
                     else "f64",
            "data": "synthetic", "config": _config(args, A),
            "iterations": st["iters"][0], "reliable_updates": st["refinements"],
            "fallbacks": st["fallbacks"], "mg_levels": st["mg_levels"],
            "true_rel_resid_l1": true_rel,
            "agreement": agreement,
            "plain_fp64_pcg": {"s_per_solve": ms_plain / 1e3, "iterations": st_plain["iters"][0]},
            "mixed_pcg": {"s_per_solve": ms_mixed / 1e3, "iterations": st_mixed["iters"][0]},
            "multigrid_jacobi_smoother": extra.get("mg_jacobi"),
            "learned_one_level": extra.get("one_level"),
            "speedup_vs_plain_fp64": ms_plain / ms_step,
            "first_call_s": first_s,
            "e2e": {"value": e2e_s / world, "unit": "s/solve",
                    "h2d_bytes_per_step": 2 * N * 8, "d2h_bytes_per_step": 2 * N * 8 + 8},
            "roofline": {"bound": "hbm", "achieved": gbs[dominant], "peak": peak, "unit": "GB/s",
                         "frac": gbs[dominant] / peak, "traffic": traffic,
                         "kernel": dominant, "alg_bytes_per_launch": alg[dominant],
                         "launch_ms": kt[dominant], "peak_kind": peak_kind},
            "kernel_gbs": {k: round(v, 1) for k, v in gbs.items()},
            "kernel_frac_of_peak": {k: round(v / peak, 3) for k, v in gbs.items()},
            "kernel_ms": {k: round(v, 4) for k, v in kt.items()},
            "vcycle_ms": vcycle_ms,
            "configs": configs,
            "cpu_baseline": cpu,
            "clocks": clocks,
            "gpu_launches": launches,
            "autotune": tune,
            "setup_s": setup_s,
        }
        print(json.dumps(line))
    s.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
