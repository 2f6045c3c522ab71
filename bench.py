#!/usr/bin/env python
"""Benchmark: solves/s to 1e-12 relative residual at 3600x2400.

Workload (one "step" = one time step of a sequence of barotropic solves):
  * operator: the 3600x2400 periodic-in-x global grid (lat in [-78, 78],
    dx = R dlon cos(lat), seeded synthetic bathymetry with ~30 % land,
    dt = 60 s), symmetric 5-point FP32 coefficients;
  * right-hand sides: a seeded field of 300 Gaussian eddies (radius
    50-150 km) advected at 0.2 m/s with slow amplitude drift, one field per
    step (the sequence workload of the learned warm start, at 3600x2400);
  * a step solves A eta_n = b_n to ||b - A eta|| / ||b|| <= 1e-12 (FP64
    residual) on the GPU.

The first --train-steps steps of the sequence are solved in FP64 (untimed);
they are the history of the timed steps and the training set of the
warm-start U-Net, which is trained on them at start-up by the library's own
BF16 forward/backward kernels (untimed).

Arms reported in one JSON line:
  value        mixed precision (FP32 PCG + FP64 refinement) from the learned
               warm start (network inference inside the timing); inputs
               resident in HBM, device-timed
  linear_mixed the same steps from linear extrapolation 2 eta[n-1] - eta[n-2]
               (no network)
  fp64_plain   the plain FP64 SEVP-PCG from a zero guess on the same steps
  e2e          the value arm through the C ABI with host buffers (b_n,
               eta_{n-1}, eta_{n-2} in, eta_n out, copies inside the timing)
  roofline     the dominant kernel (tile SEVP pass B) against measured HBM
  cpu_baseline the CPU oracle (FP64 tile-SEVP PCG, OpenMP) on the host cores

Every vector is larger than the 126 MB L2 (69 MB per FP64 field; ~1 GB of
traffic per PCG iteration), so no explicit L2 flush is done between steps.

``--impl reference`` times the CPU implementation of the method (the oracle
port; the reference's own full-width REP1 needs > 60 GB of influence
matrices at 3600 columns and its unpreconditioned BiCGSTAB needs thousands
of iterations, so neither finishes in minutes) on the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "solves/s to 1e-12 rel. residual at 3600x2400: learned+mixed vs plain FP64 SEVP"
NX, NY = 3600, 2400
# tile shape of the CPU oracle arms; the GPU arm autotunes its own (16x8 is
# what the autotuner picks on a B200 at 3600x2400)
TILE_M, TILE_H, GROWTH = 16, 8, 1e10
# --pass-b names of the library's SEVP_PASS_B_* kinds
PASS_B_KINDS = {"registers": 0, "staged": 1, "pairs": 2}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["native", "reference"], default="native")
    ap.add_argument("--nx", type=int, default=NX)
    ap.add_argument("--ny", type=int, default=NY)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--precond-fp32", type=int, default=0,
                    help="FP32 influence matrices in the inner FP32 solve of the mixed arms")
    ap.add_argument("--train-steps", type=int, default=40,
                    help="leading steps of the sequence solved in FP64 and used to train the "
                         "warm-start network (untimed)")
    ap.add_argument("--epochs", type=int, default=3)
    ap.add_argument("--coarse", type=int, default=16, choices=[1, 2, 4, 8, 16],
                    help="the network runs on the grid averaged over coarse x coarse cells")
    ap.add_argument("--tiles", default="auto",
                    help="tile shape MxH of the GPU solver, or 'auto' (measured at start-up)")
    ap.add_argument("--precond", default="auto", choices=["auto", "bj", "schwarz"],
                    help="block-Jacobi tiles, the overlapping Schwarz sweep, or 'auto' (measured)")
    ap.add_argument("--method", default="auto", choices=["auto", "pcg", "cheb"],
                    help="outer iteration of the mixed solves: PCG, the one-launch Chebyshev "
                         "iteration, or 'auto' (measured)")
    ap.add_argument("--inner-tol", default="auto",
                    help="relative reduction of each FP32 inner solve, or 'auto' (measured)")
    ap.add_argument("--influence-fp32", default="auto",
                    help="growth limit of the per-group FP32 influence data of the inner "
                         "iterations: a number, 'off', or 'auto' (measured)")
    ap.add_argument("--pass-b", default="pairs", choices=["pairs", "staged", "registers"],
                    help="kernel of the tile passes: two columns per lane, or one column per "
                         "lane with shared-memory task stages filled by tensor copies, or with "
                         "per-task register loads")
    ap.add_argument("--resume-dev", type=float, default=0.3,
                    help="largest relative distance between the recursive and the replaced "
                         "residual at which a mixed PCG run resumes (<= 0: never)")
    ap.add_argument("--no-fs", action="store_true",
                    help="skip the barotropic correction loop arm (3600x2400, 20 layers)")
    ap.add_argument("--no-ensemble", action="store_true",
                    help="skip the 64-member 720x360 ensemble arm")
    ap.add_argument("--no-learned", action="store_true",
                    help="value arm from linear extrapolation instead of the network")
    ap.add_argument("--profile", choices=["solve", "conv"], default=None,
                    help="run one small case as a profiler target and exit: 'solve' = one solve "
                         "of the global grid (--nx, --ny, --tiles, --precond, --method, "
                         "--profile-precision, --profile-max-iter); 'conv' = forward 3x3 "
                         "convolutions of the warm-start network (--conv H,W,CIN,COUT)")
    ap.add_argument("--profile-precision", type=int, default=1, choices=[0, 1])
    ap.add_argument("--profile-max-iter", type=int, default=3)
    ap.add_argument("--conv", default="600,904,256,256")
    ap.add_argument("--no-configs", action="store_true",
                    help="skip the c1 (96x96 basin), c2 (1440x720), c4 (400-step learned "
                         "sequence) and reference-call (182x92) arms")
    return ap.parse_args()


# ------------------------------------------------------------------ utils
class ClockSampler:
    """Samples nvidia-smi SM clocks and throttle reasons during a region."""

    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.rows = []
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "50"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([c.strip() for c in line.split(",")])

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            self.t.join(timeout=2)

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[0]) for r in self.rows if r[0].replace(".", "").isdigit()]
        mx = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in self.rows:
            for k, nm in enumerate(names):
                if len(r) > 4 + k and r[4 + k].lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": sorted(reasons),
                "samples": len(self.rows)}


def measured_peak_hbm():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6650.0, "fallback"


def ncu_traffic(nx, ny, tiles, kernel="passb"):
    """Per-launch DRAM bytes from the committed ncu summaries (profiles/):
    the FP32 pass-B kernel ("passb_pairs", or "passb" and "passb_staged" for
    the one-column kernels), the Schwarz stage kernel averaged over
    stages 2 and 3 ("couple") or the one-launch Chebyshev kernel ("cheb");
    None when the summary covers another grid or tile shape (they are
    3600x2400 captures with 16x6 tiles)."""
    if (nx, ny, tuple(tiles)) != (3600, 2400, (16, 6)):
        return None
    name, key = {"passb": ("tile_pass_b_3600x2400.md", "traffic_bytes_per_launch_mixed:"),
                 "passb_pairs": ("pass_b_pairs_3600x2400.md", "traffic_bytes_per_launch:"),
                 "passb_staged": ("pass_b_staged_3600x2400.md", "traffic_bytes_per_launch:"),
                 "couple": ("schwarz_stages_3600x2400.md", "traffic_bytes_per_launch_avg:"),
                 "cheb": ("cheb_3600x2400.md", "traffic_bytes_per_launch:")}[kernel]
    try:
        for line in open(os.path.join(ROOT, "profiles", name)):
            if line.startswith(key):
                return float(line.split(":")[1])
    except OSError:
        pass
    return None


def make_sequence(nx, ny, nsteps):
    from musoc_solver_b200 import problems as P

    p = P.global_grid(nx, ny, seed=11)
    rhs = [b for _, b in P.eddy_rhs(nx, ny, range(nsteps), seed=3)]
    wet = p.meta["wet"]
    rhs = [np.where(wet, b, 0.0) for b in rhs]
    return p, rhs


def dist_setup(args):
    """One process per GPU (torchrun): NCCL on the GPU box; gloo on a host
    without a GPU, where only the CPU reference arm runs."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist

        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        backend = "nccl" if torch.cuda.is_available() else "gloo"
        if backend == "nccl":
            torch.cuda.set_device(local)
        dist.init_process_group(backend, timeout=datetime.timedelta(seconds=300))
    return world, rank, local, dist


def max_over_ranks(v, dist, device):
    """The largest v over all ranks (the job's time is its slowest rank's)."""
    if dist is None:
        return v
    import torch

    t = torch.tensor([v], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ------------------------------------------------------------ CPU oracle
def cpu_solve_seconds(p, b, threads, tile_nb=None, tiles=(TILE_M, TILE_H), return_x=False):
    """One FP64 tile-SEVP PCG solve with the CPU oracle (setup excluded),
    with the same tile layout as the GPU solver."""
    os.environ["OMP_NUM_THREADS"] = str(threads)
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    from musoc_solver_b200.solver import tile_sub_blocks

    if tile_nb is None:
        tile_nb = tile_sub_blocks(p, tiles[0], tiles[1], GROWTH)
    pc = O.TilePC(p, tiles[0], tiles[1], tile_nb=tile_nb)
    t = time.perf_counter()
    x, it, rel = pc.pcg(b, tol=1e-12)
    dt = time.perf_counter() - t
    return (dt, it, rel, x) if return_x else (dt, it, rel)


def run_reference(args, world, rank):
    if rank != 0:
        return 0
    cores = os.cpu_count() or 1
    os.environ["OMP_NUM_THREADS"] = str(cores)
    p, rhs = make_sequence(args.nx, args.ny, args.warmup + args.steps)
    times, iters = [], []
    for n in range(args.warmup + args.steps):
        dt, it, rel = cpu_solve_seconds(p, rhs[n], cores)
        if n >= args.warmup:
            times.append(dt)
            iters.append(it)
    total = sum(times)
    value = len(times) / total
    line = {
        "metric": METRIC, "value": value, "unit": "solves/s", "impl": "reference",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * total / len(times), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": f"{args.nx}x{args.ny} global grid, eddy right-hand-side sequence, "
                               f"FP64 tile-SEVP PCG ({TILE_M}x{TILE_H} tiles) to 1e-12, zero guess",
                   "grid": [args.nx, args.ny], "tol": 1e-12, "l2": "inputs larger than L2"},
        "cpu_baseline": {"value": value, "unit": "solves/s", "cores": cores, "kind": "port",
                         "sample": "one full FP64 tile-SEVP PCG solve per step with the C oracle "
                                   f"(OpenMP, {cores} threads), setup excluded; mean iterations "
                                   f"{float(np.mean(iters)):.1f}"},
        "e2e": {"value": value, "unit": "solves/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


# ------------------------------------------------- CPU baselines (oracle)
def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O

    return O


def _cpu_iters_child(args):
    """One process of the all-cores baseline: `iters` PCG iterations of the
    oracle on one thread (the problem is read from .npy files)."""
    path, tiles, iters = args
    os.environ["OMP_NUM_THREADS"] = "1"
    sys.path.insert(0, ROOT)
    O = _oracle()
    from musoc_solver_b200.problems import Problem

    c = [np.load(os.path.join(path, f"{k}.npy")) for k in ("al", "ab", "ac", "ar", "at", "b")]
    nb = np.load(os.path.join(path, "tile_nb.npy"))
    p = Problem(*c, periodic=True)
    pc = O.TilePC(p, tiles[0], tiles[1], tile_nb=nb)
    t = time.perf_counter()
    pc.pcg(p.b, tol=1e-300, maxit=iters)
    return time.perf_counter() - t


def cpu_baselines(p, b, tile_nb, tiles, cores, iters_full, sample_iters=4):
    """The CPU oracle's FP64 tile-SEVP PCG on the host cores, in the two forms
    the reference's serial code allows: one solve on one thread, and one
    independent solve per core with every core busy.  Both time
    `sample_iters` PCG iterations (a bounded sample) and scale to the
    `iters_full` iterations a full solve takes."""
    import multiprocessing as mp
    import tempfile

    # each timing runs in a fresh (spawned) process whose OpenMP runtime
    # starts with one thread; this process's runtime already has all cores
    with tempfile.TemporaryDirectory() as d:
        for k, a in zip(("al", "ab", "ac", "ar", "at"), p.coeffs()):
            np.save(os.path.join(d, f"{k}.npy"), a)
        np.save(os.path.join(d, "b.npy"), b)
        np.save(os.path.join(d, "tile_nb.npy"), tile_nb)
        ctx = mp.get_context("spawn")
        job = (d, tuple(tiles), sample_iters)
        with ctx.Pool(1) as pool:
            t1 = pool.map(_cpu_iters_child, [job])[0] / sample_iters * iters_full
        with ctx.Pool(cores) as pool:
            ts = pool.map(_cpu_iters_child, [job] * cores)
    t_core = max(ts) / sample_iters * iters_full
    return {"single_thread": {"value": 1.0 / t1, "unit": "solves/s", "cores": 1,
                              "seconds_per_solve": t1},
            "one_solve_per_core": {"value": cores / t_core, "unit": "solves/s", "cores": cores,
                                   "seconds_per_solve": t_core},
            "sample": f"{sample_iters} PCG iterations per process, scaled to the {iters_full} "
                      "iterations of a full solve; setup excluded"}


# ----------------------------------------- the other configurations
def run_c1(K):
    """c1: the 96x96 closed basin.  The plain FP64 tile-SEVP PCG (24x24 tiles,
    FP64 marching sub-blocks from the growth bound) on the GPU against the
    CPU oracle of the same solve; and the reference's own direct method, REP
    on 12 row blocks of 8 rows (M/sevp.f90:335-438, influence matrices from
    PRE), as the GPU drop-in rep_ and as the CPU oracle's or_rep."""
    import ctypes as C

    import torch

    from musoc_solver_b200 import native as N, problems as P
    from musoc_solver_b200.solver import SevpSolver

    O = _oracle()
    p = P.basin(0)
    b = torch.from_numpy(p.b).cuda()
    s = SevpSolver(p, tile_m=24, tile_h=24, growth_limit=1e10)
    for _ in range(2):
        x, r = s.solve(b, precision=0)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(s.stream)
    for _ in range(K):
        x, r = s.solve(b, precision=0)
    ev1.record(s.stream)
    torch.cuda.synchronize()
    t_gpu = ev0.elapsed_time(ev1) / 1e3 / K
    pc = O.TilePC(p, 24, 24, tile_nb=s.tile_nb)
    t = time.perf_counter()
    xo, ito, relo = pc.pcg(p.b, tol=1e-12)
    t_cpu = time.perf_counter() - t
    xg = x.cpu().numpy()
    err = float(np.abs(xg - xo).max() / np.abs(xo).max())
    s.close()
    out = {"workload": "96x96 closed basin (12 seamounts, dt=60 s), FP64 tile-SEVP PCG, 24x24 "
                       "tiles, to 1e-12",
           "gpu": {"value": 1.0 / t_gpu, "unit": "solves/s", "iterations": r.iterations,
                   "rel_residual": r.rel_residual},
           "cpu_oracle": {"value": 1.0 / t_cpu, "unit": "solves/s", "iterations": ito,
                          "threads": int(os.environ["OMP_NUM_THREADS"])},
           "max_rel_err_vs_cpu_oracle": err}
    # the reference's REP on full-width row blocks
    L = N.lib()
    c = [np.ascontiguousarray(a, np.float32) for a in p.coeffs()]
    j2, i2 = p.ac.shape
    ie, _ = O.block_partition(j2, 12)
    nb = len(ie)
    rinv = np.zeros((nb, i2, i2))
    rinv1 = np.zeros((nb - 1, i2, i2))
    h = np.zeros((j2 + 2, i2 + 2))
    pp = lambda a: a.ctypes.data_as(C.c_void_p)
    ii = lambda v: C.byref(C.c_int(int(v)))
    L.sevp_set_periodic_we(0)
    L.pre_(*[pp(a) for a in c], pp(rinv), pp(rinv1), pp(h), pp(ie), ii(i2), ii(i2 + 2), ii(i2),
           ii(nb))
    f = p.b.astype(np.float32)
    d0, d1, d2 = np.zeros((nb - 1, i2)), np.zeros(i2), np.zeros(i2)
    hh = np.zeros((j2 + 2, i2 + 2))
    xr = np.zeros((j2 + 2, i2 + 2))
    L.sevp_dropin_cache(1)
    args = [pp(a) for a in c] + [pp(rinv), pp(rinv1), pp(d0), pp(d1), pp(d2), pp(f), pp(hh),
                                 pp(xr), pp(ie), ii(i2 + 2), ii(i2), ii(nb)]
    L.rep_(*args)
    t = time.perf_counter()
    for _ in range(K):
        xr[:] = 0.0
        L.rep_(*args)
    t_rep = (time.perf_counter() - t) / K
    st = L.sevp_last_status()
    L.sevp_dropin_cache(0)
    L.sevp_set_periodic_we(1)
    t = time.perf_counter()
    xro = O.rep(*c, rinv, rinv1, f, np.zeros((j2 + 2, i2 + 2)), ie)
    t_rep_cpu = time.perf_counter() - t
    res = np.linalg.norm(f - P.apply_operator(p, xr[1:-1, 1:-1])) / np.linalg.norm(f)
    out["reference_method_rep"] = {
        "method": "REP, 12 row blocks of 8 rows (influence matrices from PRE), host arrays in "
                  "and out per call, device copies of the coefficients and RINV cached",
        "gpu_dropin": {"value": 1.0 / t_rep, "unit": "solves/s", "status": st},
        "cpu_oracle": {"value": 1.0 / t_rep_cpu, "unit": "solves/s", "threads": 1},
        "bit_identical_to_cpu_oracle": bool(np.array_equal(xr, xro)),
        "rel_residual": float(res)}
    return out


def run_c2(K, tiles=(16, 6)):
    """c2: the 1440x720 periodic global grid, plain FP64 tile-SEVP PCG to
    1e-12 from zero; condition of the preconditioned operator from the
    CG-Lanczos bounds; the CPU oracle's solve and the error against it."""
    import torch

    from musoc_solver_b200 import problems as P
    from musoc_solver_b200.solver import SevpSolver

    O = _oracle()
    p = P.global_grid(1440, 720, seed=1)
    b = torch.from_numpy(p.b).cuda()
    s = SevpSolver(p, tile_m=tiles[0], tile_h=tiles[1], growth_limit=GROWTH)
    lo, hi, _ = s.estimate_bounds(b)
    for _ in range(2):
        x, r = s.solve(b, precision=0)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(s.stream)
    for _ in range(K):
        x, r = s.solve(b, precision=0)
    ev1.record(s.stream)
    torch.cuda.synchronize()
    t_gpu = ev0.elapsed_time(ev1) / 1e3 / K
    xm, rm = s.solve(b, precision=1)
    pc = O.TilePC(p, tiles[0], tiles[1], tile_nb=s.tile_nb)
    t = time.perf_counter()
    xo, ito, relo = pc.pcg(p.b, tol=1e-12)
    t_cpu = time.perf_counter() - t
    scale = np.abs(xo).max()
    out = {"workload": f"1440x720 global grid (lat +-78, ~30% land, dt=60 s), FP64 tile-SEVP "
                       f"PCG from zero to 1e-12, {tiles[0]}x{tiles[1]} tiles",
           "gpu_fp64": {"value": 1.0 / t_gpu, "unit": "solves/s", "iterations": r.iterations,
                        "rel_residual": r.rel_residual},
           "gpu_mixed": {"ms": rm.ms, "iterations": rm.iterations, "rel_residual": rm.rel_residual},
           "kappa_preconditioned": hi / lo, "lambda_min": lo, "lambda_max": hi,
           "cpu_oracle": {"value": 1.0 / t_cpu, "unit": "solves/s", "iterations": ito,
                          "threads": int(os.environ["OMP_NUM_THREADS"])},
           "max_rel_err_vs_cpu_oracle": {
               "fp64": float(np.abs(x.cpu().numpy() - xo).max() / scale),
               "mixed": float(np.abs(xm.cpu().numpy() - xo).max() / scale)}}
    s.close()
    return out


def run_reference_call(K):
    """The reference's solver call at its own 182x92 grid: FS_SOLVER's
    FL_EVP_STP = 0 path (M/fs_GLOBAL.f90:1852-1853), REP1 on 15 row blocks
    then p_bicgstab_le, on the reference's test stencil
    (P/prep_GLOBAL.f90:246-261, AC shifted by 0.01 so that the system is not
    singular) with a REAL*4 right-hand side: the GPU drop-ins rep1_ and
    p_bicgstab_le_ (host arrays, device copies of RINV cached) against the
    CPU oracle's or_rep1 and or_bicgstab_le on one thread; and the fast
    drop-in p_sevp_pcg_ with the same argument list, to 1e-12 relative."""
    import ctypes as C

    from musoc_solver_b200 import native as N, problems as P

    O = _oracle()
    L = N.lib()
    p = P.idealised(180, 90)
    p.ac[:] += np.float32(0.01)
    c = [np.ascontiguousarray(a, np.float32) for a in p.coeffs()]
    j2, i2 = p.ac.shape
    rng = np.random.default_rng(5)
    f = rng.standard_normal((j2, i2)).astype(np.float32)
    ie, _ = O.block_partition(j2, 15)
    nb = len(ie)
    pp = lambda a: a.ctypes.data_as(C.c_void_p)
    ii = lambda v: C.byref(C.c_int(int(v)))
    rinv = np.zeros((nb, i2, i2))
    rinv1 = np.zeros((nb - 1, i2, i2))
    h = np.zeros((j2 + 2, i2 + 2))
    L.sevp_set_periodic_we(1)
    L.pre1_(*[pp(a) for a in c], pp(rinv), pp(rinv1), pp(h), pp(ie), ii(i2 + 2), ii(i2), ii(nb))
    d0, d1, d2 = np.zeros((nb - 1, i2)), np.zeros(i2), np.zeros(i2)
    hh = np.zeros((j2 + 2, i2 + 2))
    x = np.zeros((j2 + 2, i2 + 2))
    L.sevp_dropin_cache(1)

    def gpu_rep1():
        x[:] = 0.0
        L.rep1_(*[pp(a) for a in c], pp(rinv), pp(rinv1), pp(d0), pp(d1), pp(d2), pp(f), pp(hh),
                pp(x), pp(ie), ii(i2 + 2), ii(i2), ii(nb))

    def gpu_bicg():
        xb = np.zeros((j2 + 2, i2 + 2))
        L.p_bicgstab_le_(*[pp(a) for a in c], pp(f), pp(xb), *[pp(a) for a in c], ii(i2), ii(j2))
        return xb

    def gpu_fast():
        xf = np.zeros((j2 + 2, i2 + 2))
        L.p_sevp_pcg_(*[pp(a) for a in c], pp(f), pp(xf), *[pp(a) for a in c], ii(i2), ii(j2))
        return xf

    def timed(fn, n):
        fn()
        t = time.perf_counter()
        for _ in range(n):
            out = fn()
        return (time.perf_counter() - t) / n, out

    t_rep1, _ = timed(gpu_rep1, K)
    xrep = x.copy()
    t_bicg, xb = timed(gpu_bicg, max(1, K // 4))
    o = N.FsOptions()
    L.sevp_fs_default_options(C.byref(o))
    L.sevp_fs_set_options(C.byref(o))
    t_fast, xf = timed(gpu_fast, K)
    rep = N.Report()
    L.sevp_fs_last_report(C.byref(rep))
    L.sevp_dropin_cache(0)
    L.sevp_fs_release()
    t = time.perf_counter()
    xro = O.rep1(*c, rinv, rinv1, f, np.zeros((j2 + 2, i2 + 2)), ie)
    t_rep1_cpu = time.perf_counter() - t
    t = time.perf_counter()
    xbo, itbo, resbo = O.bicgstab(*c, f, np.zeros((j2 + 2, i2 + 2)))
    t_bicg_cpu = time.perf_counter() - t
    rel = lambda xx: float(np.linalg.norm(f - P.apply_operator(p, xx[1:-1, 1:-1]))
                           / np.linalg.norm(f))
    return {"workload": "182x92 (I0 x J0), the reference's test stencil (AC + 0.01), REAL*4 "
                        "right-hand side N(0,1); FS_SOLVER FL_EVP_STP=0: REP1 (15 row blocks) "
                        "then p_bicgstab_le (stop: sqrt(r.r) <= 1e-8)",
            "rep1": {"gpu_dropin": {"value": 1.0 / t_rep1, "unit": "calls/s"},
                     "cpu_oracle": {"value": 1.0 / t_rep1_cpu, "unit": "calls/s", "threads": 1},
                     "bit_identical_to_cpu_oracle": bool(np.array_equal(xrep, xro)),
                     "rel_residual": rel(xrep)},
            "p_bicgstab_le": {"gpu_dropin": {"value": 1.0 / t_bicg, "unit": "calls/s"},
                              "cpu_oracle": {"value": 1.0 / t_bicg_cpu, "unit": "calls/s",
                                             "threads": 1, "iterations": itbo},
                              "rel_residual": rel(xb),
                              "max_abs_diff_vs_cpu_oracle": float(np.abs(xb - xbo).max())},
            "p_sevp_pcg": {"gpu_dropin": {"value": 1.0 / t_fast, "unit": "calls/s",
                                          "iterations": rep.iterations},
                           "rel_residual": rel(xf),
                           "max_rel_err_vs_rep1_cpu_oracle":
                               float(np.abs(xf - xro)[1:-1, 1:-1].max()
                                     / np.abs(xro[1:-1, 1:-1]).max())}}


def run_c4(steps=400, train_steps=300, coarse=4, epochs=3, tiles=(16, 8)):
    """c4: the learned warm start on a 400-step 1440x720 eddy sequence: FP64
    solves of every step (the training data), the U-Net trained on steps
    2..299 and tested on 302..399 with iterations and device time (guess +
    mixed solve to 1e-12) from the zero, previous, linear and learned
    guesses."""
    import torch

    from musoc_solver_b200 import problems as P
    from musoc_solver_b200.solver import SevpSolver
    from musoc_solver_b200.warmstart import LearnedWarmStart, evaluate, solve_sequence, train

    t0 = time.perf_counter()
    p = P.global_grid(1440, 720, seed=1)
    wet = p.meta["wet"]
    rhs = [torch.from_numpy(np.where(wet, b, 0.0)).cuda()
           for _, b in P.eddy_rhs(1440, 720, range(steps), seed=3)]
    s = SevpSolver(p, tile_m=tiles[0], tile_h=tiles[1], growth_limit=GROWTH)
    etas = solve_sequence(s, rhs)
    torch.cuda.synchronize()
    t_seq = time.perf_counter() - t0
    train_idx = list(range(2, train_steps))
    test_idx = list(range(train_steps + 2, steps))
    t1 = time.perf_counter()
    w = LearnedWarmStart.create(s, seed=0, train=True, coarse=coarse)
    losses = train(w, etas, rhs, train_idx, epochs=epochs, lr=2e-3, lr_final=2e-4)
    torch.cuda.synchronize()
    t_train = time.perf_counter() - t1
    w = w.inference_copy()
    x = torch.zeros_like(etas[0])
    gain = []
    for n in test_idx:
        w.predict(etas[n - 1], etas[n - 2], rhs[n], x)
        gain.append(float((w.e + w.m - etas[n]).norm() / (x - etas[n]).norm()))
    w.attach()
    res = evaluate(s, w, etas, rhs, test_idx)
    w.close()
    s.close()
    return {"workload": f"1440x720 global grid, {steps}-step eddy sequence (300 eddies, 0.2 m/s), "
                        f"train steps 2-{train_steps - 1}, test {train_steps + 2}-{steps - 1}; "
                        f"network on the 1/{coarse} grid; mixed solve to 1e-12, "
                        f"{tiles[0]}x{tiles[1]} tiles",
            "fp64_sequence_seconds": t_seq, "train_seconds": t_train, "epochs": epochs,
            "loss_first_last": [losses[0][1], losses[-1][1]],
            "guess_error_ratio_without_over_with_network": float(np.median(gain)),
            "test": res}


# --------------------------------------------------------------- ensemble
def run_ensemble(K, W, members=64, nx=720, ny=360, schwarz=False, inner_tol=1e-5,
                 oracle_check=True):
    """64 members x 720x360 (independently perturbed depths and right-hand
    sides) stacked into one system: every kernel launch covers all members."""
    import torch

    from musoc_solver_b200 import problems as P
    from musoc_solver_b200.ensemble import EnsembleSolver

    t0 = time.perf_counter()
    ms = P.ensemble(members=members, nx=nx, ny=ny, seed=5)
    e = EnsembleSolver(ms)
    e_th = e.solver.tile_h  # the oracle check uses the same tiles
    setup_s = time.perf_counter() - t0
    b = e.rhs()
    stream = e.solver.stream
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    out = {"workload": f"{members} members x {nx}x{ny}, +-5% depth noise, own right-hand sides, "
                       f"stacked ({e.problem.nx}x{e.problem.ny}), tiles {e.solver.tile_m}x{e.solver.tile_h}",
           "setup_seconds": setup_s}
    from musoc_solver_b200 import native as N

    # (name, precision, Schwarz, one-launch Chebyshev iteration)
    arms = [("mixed", 1, False, False), ("fp64", 0, False, False), ("mixed_cheb", 1, False, True)]
    if schwarz:
        arms += [("mixed_schwarz", 1, True, False), ("fp64_schwarz", 0, True, False)]
    for name, prec, sw, cheb in arms:
        if sw != bool(e.solver.schwarz_shift):
            e.solver.set_schwarz(-1 if sw else 0)
        if cheb:
            # spectrum bounds of the stacked operator (set-up, untimed)
            e.solver.chebyshev_setup(b)
        e.solver.set_method(N.METHOD_CHEB if cheb else N.METHOD_PCG)
        x = torch.zeros_like(b)
        tol_stack = e.stacked_tol(b)
        for _ in range(W):
            e.solve(b, x=x, precision=prec, inner_tol=inner_tol, residuals=False,
                    tol_stack=tol_stack, x_is_guess=False)
        torch.cuda.synchronize()
        # the timed solves: every launch is the library's (from zero into x,
        # the per-member residuals measured after the timing)
        ev0.record(stream)
        res = None
        for _ in range(K):
            x, res, _ = e.solve(b, x=x, precision=prec, inner_tol=inner_tol, residuals=False,
                                tol_stack=tol_stack, x_is_guess=False)
        ev1.record(stream)
        torch.cuda.synchronize()
        t = ev0.elapsed_time(ev1) / 1e3
        rel = e.member_residuals(b, x)
        out[name] = {"value": members * K / t, "unit": "member solves/s", "ms_per_ensemble": 1e3 * t / K,
                     "iterations": res.iterations, "max_member_rel_residual": float(rel.max())}
        if cheb:
            out[name]["launches_per_iteration"] = 1
            e.solver.set_method(N.METHOD_PCG)
        if name == "mixed":
            xm = x.clone()
        if name == "fp64":
            x64 = x.clone()
    # per-member error of the mixed solve against the FP64 solve on the GPU
    d = (xm - x64).reshape(members, -1).abs().amax(dim=1)
    ref = x64.reshape(members, -1).abs().amax(dim=1)
    out["mixed"]["max_member_rel_err_vs_fp64"] = float((d / ref).max())
    e.close()
    # and every member of both solves against the CPU oracle's FP64 PCG of
    # that member alone
    if oracle_check:
        from musoc_solver_b200.solver import tile_sub_blocks

        O = _oracle()
        xm_h = xm.reshape(members, ny, nx).cpu().numpy()
        x64_h = x64.reshape(members, ny, nx).cpu().numpy()
        errs_m, errs_64, t0 = [], [], time.perf_counter()
        for k, m in enumerate(ms):
            th = e_th
            pc = O.TilePC(m, 16, th, tile_nb=tile_sub_blocks(m, 16, th, GROWTH))
            xo, _, relo = pc.pcg(m.b, tol=1e-12)
            sc = np.abs(xo).max()
            errs_m.append(float(np.abs(xm_h[k] - xo).max() / sc))
            errs_64.append(float(np.abs(x64_h[k] - xo).max() / sc))
        out["max_member_rel_err_vs_cpu_oracle"] = {"mixed": max(errs_m), "fp64": max(errs_64),
                                                   "members": members,
                                                   "oracle_seconds": time.perf_counter() - t0}
    return out


# ------------------------------------------------ barotropic correction loop
def run_fs(nx, ny, k1, tiles, passes=3, peak=None, schwarz=False, inner_tol=1e-5):
    """The FS barotropic correction (ITMASK loop) on a layered state: one
    pass = land masking, continuity right-hand side, mixed solve, P0 and
    velocity correction of every layer."""
    import torch

    from musoc_solver_b200 import problems as P
    from musoc_solver_b200.barotropic import BarotropicCorrection

    st = P.fs_state(nx, ny, k1, seed=7)
    bc = BarotropicCorrection(st, tile_m=tiles[0], tile_h=tiles[1], schwarz=schwarz)
    u, v, p0, scr = bc.upload()
    stream = bc.solver.stream
    bc.run(u, v, p0, scr, tolerance=0.0, mxmask=1, inner_tol=inner_tol)  # warm-up pass
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    ev0.record(stream)
    n_pass, vmax, iters = bc.run(u, v, p0, scr, tolerance=0.0, mxmask=passes, inner_tol=inner_tol)
    ev1.record(stream)
    torch.cuda.synchronize()
    t_loop = ev0.elapsed_time(ev1) / n_pass

    def time_ms(fn, reps=5):
        fn()
        torch.cuda.synchronize()
        ev0.record(stream)
        for _ in range(reps):
            fn()
        ev1.record(stream)
        torch.cuda.synchronize()
        return ev0.elapsed_time(ev1) / reps

    n = nx * ny
    t_rhs = time_ms(lambda: bc.rhs(u, v, b=bc.b))
    t_cor = time_ms(lambda: bc.correct(bc.x, u, v, p0, scr))
    # algorithmic bytes: rhs reads U and V of every layer, writes b; the
    # correction reads X and masks, reads and writes U, V, P0 and 4 SCR planes
    b_rhs = n * (8 * k1 + 8)
    b_cor = n * (8 + 12 * k1 + 8 + 8 + 16)
    gbs = lambda b, ms: b / (ms * 1e-3) / 1e9
    out = {"workload": f"{nx}x{ny} interior, {k1} layers, land masks from the synthetic depth; "
                       f"mixed solve to 1e-12, tiles {tiles[0]}x{tiles[1]}"
                       f"{', Schwarz preconditioner' if schwarz else ''}",
           "ms_per_pass": t_loop, "passes": n_pass, "pcg_iterations": iters,
           "land_velocity_after": vmax,
           "rhs_ms": t_rhs, "rhs_gbs": gbs(b_rhs, t_rhs), "correct_ms": t_cor,
           "correct_gbs": gbs(b_cor, t_cor)}
    if peak:
        out["rhs_frac"] = gbs(b_rhs, t_rhs) / peak
        out["correct_frac"] = gbs(b_cor, t_cor) / peak
    bc.close()
    return out


# ---------------------------------------------------------------- native
def run_native(args, world, rank, local, dist):
    import torch

    from musoc_solver_b200 import build, native as N
    from musoc_solver_b200.solver import SevpSolver

    build.build()
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)
    K, W = args.steps, args.warmup

    T = max(args.train_steps, 4)
    nsteps = T + W + K
    p, rhs = make_sequence(args.nx, args.ny, nsteps)
    n = p.nx * p.ny
    # the leading T steps: FP64 solves from linear extrapolation (untimed);
    # they are the history of the timed steps and the network's training set
    # (block-Jacobi 16x6 tiles; the solutions do not depend on the solver
    # configuration beyond the 1e-12 tolerance)
    from musoc_solver_b200.autotune import CANDIDATES, SCHWARZ_MAX_ROWS, autotune
    from musoc_solver_b200.warmstart import LearnedWarmStart, solve_sequence, train

    b_dev = [torch.from_numpy(b).to(dev) for b in rhs]
    base = SevpSolver(p, tile_m=16, tile_h=6, growth_limit=GROWTH, precond_fp32=args.precond_fp32)
    eta = solve_sequence(base, b_dev[:T])

    # tile shape, preconditioner and inner tolerance: measured (untimed) on
    # step T-1 from the linear extrapolation of its history, the warm start
    # the timed arms use, unless all three are given
    tune_table = None
    cands = CANDIDATES if args.tiles == "auto" else (
        tuple(int(v) for v in args.tiles.lower().split("x")),)
    sw_opts = {"auto": (False, True), "bj": (False,), "schwarz": (True,)}[args.precond]
    itols = (1e-3, 1e-4, 1e-5) if args.inner_tol == "auto" else (float(args.inner_tol),)
    methods = {"auto": (N.METHOD_PCG, N.METHOD_CHEB), "pcg": (N.METHOD_PCG,),
               "cheb": (N.METHOD_CHEB,)}[args.method]
    if len(cands) * len(sw_opts) * len(itols) * len(methods) > 1:
        best, tune_table = autotune(p, b_dev[T - 1], candidates=cands, precision=1,
                                    growth_limit=GROWTH, schwarz=sw_opts, inner_tols=itols,
                                    history=(eta[T - 2], eta[T - 3]), methods=methods)
        tiles, use_sw, itol = (best["tile_m"], best["tile_h"]), best["schwarz"], best["inner_tol"]
        method = best["method"]
    else:
        tiles, use_sw, itol, method = cands[0], sw_opts[0], itols[0], methods[0]
    if dist is not None:
        # every rank runs the same arms (and so the same collectives): rank
        # 0's choice holds for all
        choice = [(tuple(tiles), bool(use_sw), float(itol), int(method))]
        dist.broadcast_object_list(choice, src=0)
        tiles, use_sw, itol, method = choice[0]
    if use_sw and tiles[1] > SCHWARZ_MAX_ROWS:
        raise SystemExit(f"the Schwarz preconditioner needs tiles of at most {SCHWARZ_MAX_ROWS} rows")
    if tuple(tiles) == (16, 6) and not use_sw:
        solver = base
    else:
        base.close()
        solver = SevpSolver(p, tile_m=tiles[0], tile_h=tiles[1], growth_limit=GROWTH,
                            precond_fp32=args.precond_fp32, schwarz=use_sw)
    solver.set_pass_b_kernel(PASS_B_KINDS[args.pass_b])
    solver.set_resume_check(args.resume_dev)
    stream = solver.stream
    cheb_bounds = None
    if method == N.METHOD_CHEB:
        # spectrum bounds of the operator's set-up (untimed, like the
        # influence data)
        cheb_bounds = solver.chebyshev_setup(b_dev[T - 1])
    solver.set_method(method)
    torch.cuda.synchronize()

    # per-group FP32 influence data of the inner iterations (tile passes):
    # growth limit measured (untimed) on the same warm-start step, unless given
    mix_limit, mix_table = 0.0, None
    if args.influence_fp32 == "auto" and not args.precond_fp32:
        mix_table, xw = {}, torch.zeros_like(eta[0])
        for lim in (0.0, 1e3, 1e4, 1e5, 1e6):
            solver.set_influence_fp32(lim)
            ts, ok = [], True
            for _ in range(3):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                _, r = solver.solve_step(b_dev[T - 1], eta[T - 2], eta[T - 3], xw,
                                         guess=N.GUESS_LINEAR, precision=1, inner_tol=itol)
                torch.cuda.synchronize()
                ts.append(time.perf_counter() - t0)
                ok = ok and r.status == 0
            if ok:
                mix_table[f"{lim:g}" if lim else "off"] = round(min(ts[1:]) * 1e3, 3)
                if min(ts[1:]) * 1e3 <= min(mix_table.values()):
                    mix_limit = lim
    elif args.influence_fp32 not in ("auto", "off"):
        mix_limit = float(args.influence_fp32)
    if dist is not None:
        choice = [float(mix_limit)]
        dist.broadcast_object_list(choice, src=0)
        mix_limit = choice[0]
    solver.set_influence_fp32(mix_limit)
    mix_groups = solver.influence_fp32_groups()
    torch.cuda.synchronize()

    eta += [torch.zeros_like(eta[0]) for _ in range(W + K)]
    guess_mode, guess_name = N.GUESS_LINEAR, "linear extrapolation 2*eta[n-1]-eta[n-2]"
    warm, train_info = None, None
    if not args.no_learned:
        t0 = time.perf_counter()
        trainer = LearnedWarmStart.create(solver, seed=0, train=True, coarse=args.coarse)
        losses = train(trainer, eta, b_dev, list(range(2, T)), epochs=args.epochs, lr=2e-3,
                       lr_final=2e-4)
        warm = trainer.inference_copy()
        del trainer
        torch.cuda.synchronize()
        warm.attach(solver)
        guess_mode = N.GUESS_LEARNED
        guess_name = (f"learned: U-Net (4 levels, 32 base channels, BF16) on the "
                      f"{warm.net.H}x{warm.net.W} grid ({args.coarse}x{args.coarse} averages), "
                      "correction added to 2*eta[n-1]-eta[n-2] + one tile-SEVP solve")
        train_info = {"steps": T - 2, "epochs": args.epochs, "seconds": time.perf_counter() - t0,
                      "loss_first": losses[0][1], "loss_last": losses[-1][1],
                      "network_grid": [warm.net.W, warm.net.H]}

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()


    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    timed = range(T + W, T + W + K)

    def run_arm(mode, hist):
        """Warm-up and timed steps of a sequence arm; hist holds the solutions."""
        for k in range(T, T + W):
            solver.solve_step(b_dev[k], hist[k - 1], hist[k - 2], hist[k], guess=mode, precision=1,
                              inner_tol=itol)
        barrier()
        reps = []
        l0 = solver.launches()
        ev0.record(stream)
        for k in timed:
            _, r = solver.solve_step(b_dev[k], hist[k - 1], hist[k - 2], hist[k], guess=mode,
                                     precision=1, inner_tol=itol)
            reps.append(r)
        ev1.record(stream)
        torch.cuda.synchronize()
        return max_over_ranks(ev0.elapsed_time(ev1) / 1e3, dist, dev), reps, solver.launches() - l0

    # ---- value arm: mixed precision + warm start, device-resident inputs
    with ClockSampler(local) as clk:
        t_value, reps, launches_value = run_arm(guess_mode, eta)
    # per-kernel device times of the same steps, from an untimed replay with
    # CUDA events around every launch (the events and the direct launches
    # they need would slow the timed arm)
    solver.profile(True)
    run_arm(guess_mode, eta)
    prof = solver.profile_read()
    solver.profile(False)
    relres = [r.rel_residual for r in reps]
    status = [r.status for r in reps]

    # ---- the same sequence from linear extrapolation (no network)
    eta_lin = eta[:T] + [torch.zeros_like(eta[0]) for _ in range(W + K)]
    t_lin, reps_lin, _ = run_arm(N.GUESS_LINEAR, eta_lin)
    x_lin0 = eta_lin[timed[0]].cpu().numpy()
    del eta_lin

    # error of the value arm against an FP64 solve of the same steps (the
    # FP64 solve of the first timed step is kept for the CPU-oracle check)
    ref_x = torch.zeros_like(eta[0])
    errs = []
    x64_0 = None
    for k in (timed[0], timed[-1]):
        solver.solve(b_dev[k], x=ref_x.zero_(), precision=0)
        errs.append(float((eta[k] - ref_x).abs().max() / ref_x.abs().max()))
        if x64_0 is None:
            x64_0 = ref_x.cpu().numpy()

    # ---- plain FP64 SEVP-PCG from a zero guess (block-Jacobi tiles)
    def fp64_zero_arm():
        xz = torch.zeros_like(eta[0])
        for k in range(T, T + W):
            solver.solve(b_dev[k], x=xz, precision=0, x_is_guess=False)
        barrier()
        ev0.record(stream)
        its = []
        for k in timed:
            _, r = solver.solve(b_dev[k], x=xz, precision=0, x_is_guess=False)
            its.append(r.iterations)
        ev1.record(stream)
        torch.cuda.synchronize()
        return max_over_ranks(ev0.elapsed_time(ev1) / 1e3, dist, dev), its

    if use_sw:
        solver.set_schwarz(0)
    t_fp64, it64 = fp64_zero_arm()
    fp64_sw = None
    if use_sw:
        solver.set_schwarz(-1)
        t_sw, it_sw = fp64_zero_arm()
        fp64_sw = {"value": world * K / t_sw, "unit": "solves/s", "ms_per_step": 1e3 * t_sw / K,
                   "mean_iterations": float(np.mean(it_sw))}
    xz = torch.zeros_like(eta[0])

    # ---- mixed precision from a zero guess (isolates the precision gain)
    barrier()
    ev0.record(stream)
    itmz = []
    for k in timed:
        _, r = solver.solve(b_dev[k], x=xz, precision=1, inner_tol=itol, x_is_guess=False)
        itmz.append(r.iterations)
    ev1.record(stream)
    torch.cuda.synchronize()
    t_mixed0 = max_over_ranks(ev0.elapsed_time(ev1) / 1e3, dist, dev)

    # ---- e2e: the same value arm through the C ABI with host buffers.
    #      The context keeps the last two solutions in device memory, so a
    #      step copies b in and x out (pinned buffers).  Headline: the
    #      asynchronous steps (step n+1's b prefetched during step n's
    #      solve, x copied out on a copy stream); beside it the synchronous
    #      step, and the steps with the history copied in every step.
    pin = lambda a: torch.from_numpy(a).pin_memory().numpy()
    b_host = {k: pin(rhs[k]) for k in range(T, T + W + K)}
    eta_host = {k: pin(np.zeros((p.ny, p.nx))) for k in range(T - 2, T + W + K)}
    for k in (T - 2, T - 1):
        eta_host[k][:] = eta[k].cpu().numpy()
    solver.step_history(eta_host[T - 1], eta_host[T - 2])
    for k in range(T, T + W):
        solver.step_submit(b_host[k], eta_host[k], guess=guess_mode, precision=1, inner_tol=itol)
    solver.step_wait()
    barrier()
    t0 = time.perf_counter()
    l1 = solver.launches()
    solver.step_prefetch(b_host[timed[0]])
    for k in timed:
        if k + 1 in timed:
            solver.step_prefetch(b_host[k + 1])
        solver.step_submit(b_host[k], eta_host[k], guess=guess_mode, precision=1, inner_tol=itol)
    solver.step_wait()
    torch.cuda.synchronize()
    t_e2e = max_over_ranks(time.perf_counter() - t0, dist, dev)
    launches_e2e = solver.launches() - l1
    h2d = 8 * n
    d2h = 8 * n
    # the synchronous step (history on the device, copies not overlapped)
    solver.step_history(eta_host[timed[0] - 1], eta_host[timed[0] - 2])
    barrier()
    t0 = time.perf_counter()
    for k in timed:
        solver.step_host(b_host[k], eta_host[k], guess=guess_mode, precision=1, inner_tol=itol)
    torch.cuda.synchronize()
    t_e2e_sync = max_over_ranks(time.perf_counter() - t0, dist, dev)
    barrier()
    t0 = time.perf_counter()
    for k in timed:
        solver.solve_step_host(b_host[k], eta_host[k - 1], eta_host[k - 2], eta_host[k],
                               guess=guess_mode, precision=1, inner_tol=itol)
    torch.cuda.synchronize()
    t_e2e_hist = max_over_ranks(time.perf_counter() - t0, dist, dev)
    h2d_hist = 8 * n * (3 if guess_mode in (N.GUESS_LINEAR, N.GUESS_LEARNED) else 2)

    # ---- roofline of the dominant kernel (FP32 vectors): pass B with the
    #      block-Jacobi preconditioner, the Schwarz stage kernel otherwise
    peak, peak_kind = measured_peak_hbm()
    tile_ms, tile_n = prof["tile"]
    cpl_ms, cpl_n = prof["couple"]
    ncoef = 3 if solver.symmetric else 5
    scale = 0.5 if args.precond_fp32 else 1.0
    # influence bytes one block-Jacobi tile pass reads (per-group precision
    # when it is on)
    infl_a = int(solver.influence_bytes() * scale) if args.precond_fp32 else mix_groups[2]
    infl_b = int(solver.schwarz_influence_bytes() * scale)
    # pass B: r,q in; r,z out (z1 with the Schwarz preconditioner);
    # coefficient planes; influence data
    b_passb = n * (2 * 4 + 2 * 4 + 4 * ncoef) + infl_a
    # Schwarz stages, per launch averaged over stage 2 (w in, z2 out) and
    # stage 3 (w, z1, r in, z out): halo rows of w (2 per tile row) and of
    # AT (symmetric storage), coefficient planes, the tiling's influence data
    halo = (2 * 4 + (4 if solver.symmetric else 0)) / tiles[1]
    b_stage2 = n * (4 + 4 + halo + 4 * ncoef) + infl_b
    b_stage3 = n * (4 + 4 + 4 + 4 + halo + 4 * ncoef) + infl_a
    b_couple = 0.5 * (b_stage2 + b_stage3)
    # one Chebyshev launch: d (own rows, halo from L2), x, r in; x, r, d out;
    # coefficient planes; influence data
    b_cheb = n * (4 * 3 + 4 * 3 + 4 * ncoef) + infl_a
    short_tiles = tiles[1] <= 6  # FP32 vectors with tiles up to 6 rows run the short-tile kernel
    kind = solver.pass_b_kernel_used()
    staged = kind == N.PASS_B_STAGED
    if kind == N.PASS_B_PAIRS:
        passb_name = "k_tile_pair<float, update, dots> (PCG pass B, two columns per lane)"
    elif staged:
        passb_name = "k_pass_b_tma (PCG pass B, tensor-copied task stages)"
    else:
        passb_name = ("k_tile_short<float, update, dots>" if short_tiles
                      else "k_tile_apply<float, update, dots>") + " (PCG pass B)"
    if method == N.METHOD_CHEB:
        dom_name = "k_cheb<float> (one-launch Chebyshev iteration)"
        bytes_per_launch, avg_s, dom_n = b_cheb, tile_ms / 1e3 / max(tile_n, 1), tile_n
        traffic = ncu_traffic(p.nx, p.ny, tiles, "cheb")
    elif use_sw and cpl_n:
        dom_name = "k_tile_couple<float> (Schwarz stages 2 and 3, averaged per launch)"
        bytes_per_launch, avg_s, dom_n = b_couple, cpl_ms / 1e3 / cpl_n, cpl_n
        traffic = ncu_traffic(p.nx, p.ny, tiles, "couple")
    else:
        dom_name = passb_name
        bytes_per_launch, avg_s, dom_n = b_passb, tile_ms / 1e3 / max(tile_n, 1), tile_n
        traffic = ncu_traffic(p.nx, p.ny, tiles,
                              {N.PASS_B_PAIRS: "passb_pairs",
                               N.PASS_B_STAGED: "passb_staged"}.get(kind, "passb"))
    achieved = bytes_per_launch / avg_s / 1e9 if dom_n else None

    # ---- 64-member ensemble (720x360 each), every launch over all members
    ens = None
    if not args.no_ensemble:
        ens = run_ensemble(max(2, K // 2), max(1, min(W, 2)), schwarz=True, inner_tol=itol)

    # ---- the barotropic correction loop around the solve (FS ITMASK loop)
    fs = None
    if not args.no_fs:
        fs = run_fs(p.nx, p.ny, 20, tiles, peak=peak, schwarz=use_sw, inner_tol=itol)

    # ---- the other configurations (rank 0 at N = 1; no collectives)
    c1 = c2 = c4 = ref_call = None
    if rank == 0 and world == 1 and not args.no_configs:
        c1 = run_c1(max(K, 10))
        c2 = run_c2(max(2, K // 2))
        ref_call = run_reference_call(max(4, K // 2))
        if not args.no_learned:
            c4 = run_c4()

    # ---- CPU baseline and the error against the CPU oracle (rank 0 at N = 1)
    cpu, cpu_forms, oracle_err = None, None, None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cores = os.cpu_count() or 1
        k0 = timed[0]
        dt, itc, relc, xo = cpu_solve_seconds(p, rhs[k0], cores, solver.tile_nb, tiles,
                                              return_x=True)
        cpu = {"value": 1.0 / dt, "unit": "solves/s", "cores": cores, "kind": "port",
               "sample": f"one full FP64 tile-SEVP PCG solve of step {k0} with the C oracle "
                         f"(OpenMP, {cores} threads, {itc} iterations, rel. residual {relc:.2e}), "
                         "setup excluded"}
        cpu_forms = cpu_baselines(p, rhs[k0], solver.tile_nb, tiles, cores, itc)
        sc = float(np.abs(xo).max())

        def err(xg):
            d = float(np.abs(xg - xo).max())
            return {"max_abs_deta": d, "max_rel_deta": d / sc}

        oracle_err = {"step": k0, "oracle": "C oracle FP64 tile-SEVP PCG to 1e-12",
                      "value_arm": err(eta[k0].cpu().numpy()), "linear_mixed": err(x_lin0),
                      "fp64_plain": err(x64_0)}

    value = world * K / t_value
    line = {
        "metric": METRIC,
        "value": value,
        "unit": "solves/s",
        "n_gpus": world,
        "steps": K,
        "warmup": W,
        "ms_per_step": 1e3 * t_value / K,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32+f64",
        "data": "synthetic",
        "config": {
            "workload": f"{p.nx}x{p.ny} global grid (lat +-78, ~30% land, dt=60 s), eddy "
                        "right-hand-side sequence; mixed FP32 tile-SEVP PCG + FP64 iterative "
                        f"refinement to 1e-12 from warm start: {guess_name}",
            "grid": [p.nx, p.ny], "tiles": list(tiles),
            "preconditioner": (f"overlapping Schwarz, second tiling shifted by "
                               f"{solver.schwarz_shift} columns" if use_sw else "block-Jacobi tiles"),
            "inner_tol": itol,
            "outer_iteration": "one-launch Chebyshev" if method == N.METHOD_CHEB else "PCG",
            "chebyshev_bounds": cheb_bounds,
            "tile_autotune": None if tune_table is None else
            {f"{r['tile_m']}x{r['tile_h']}{' schwarz' if r['schwarz'] else ''}"
             f"{' cheb' if r['method'] == N.METHOD_CHEB else ''} itol={r['inner_tol']:g}":
             round(r["ms"], 2) for r in tune_table},
            "tile_autotune_workload": "one warm-start step (linear extrapolation), mixed solve",
            "marching_growth_limit": GROWTH,
            "coefficient_planes": 3 if solver.symmetric else 5,
            "influence_fp32_in_inner_solve": bool(args.precond_fp32),
            "resume_check_max_rel_dev": args.resume_dev,
            "pass_b_kernel": {N.PASS_B_PAIRS: "pairs (two columns per lane)",
                              N.PASS_B_STAGED: "staged (tensor-copied task stages)",
                              N.PASS_B_REGISTERS: "registers"}.get(solver.pass_b_kernel_used(),
                                                                    "none"),
            "influence_fp32_growth_limit": mix_limit or None,
            "influence_fp32_groups": [mix_groups[0], mix_groups[1]],
            "influence_bytes_per_tile_pass": mix_groups[2],
            "influence_fp32_autotune_ms": mix_table,
            "tol": 1e-12, "parallelism": f"replicas x{world}",
            "l2": "inputs larger than L2 (69 MB per FP64 field), no flush",
        },
        "fp64_schwarz_zero_guess": fp64_sw,
        "mixed_zero_guess": {"value": world * K / t_mixed0, "unit": "solves/s",
                             "mean_iterations": float(np.mean(itmz))},
        "warm_start_training": train_info,
        "e2e": {"value": world * K / t_e2e, "unit": "solves/s", "h2d_bytes_per_step": h2d,
                "d2h_bytes_per_step": d2h,
                "api": "sevp_step_prefetch / sevp_step_submit / sevp_step_wait (history of the "
                       "two previous solutions held in HBM; copies overlapped with the solves)"},
        "e2e_step_host": {"value": world * K / t_e2e_sync, "unit": "solves/s",
                          "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                          "api": "sevp_step_host (history in HBM, copies not overlapped)"},
        "e2e_history_from_host": {"value": world * K / t_e2e_hist, "unit": "solves/s",
                                  "h2d_bytes_per_step": h2d_hist, "d2h_bytes_per_step": d2h,
                                  "api": "sevp_solve_step_host (b, eta1, eta2 copied in)"},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": (achieved / peak) if achieved else None, "traffic": traffic,
                     "kernel": dom_name,
                     "algorithmic_bytes_per_launch": bytes_per_launch,
                     "avg_launch_ms": avg_s * 1e3, "launches": dom_n,
                     "peak_source": f"{peak_kind} copy bandwidth (MEASURED_PEAKS.json hbm_gbs)"},
        "kernels": {"tile_pass_b" if method != N.METHOD_CHEB else "chebyshev": {
                                    "launches": tile_n,
                                    "avg_ms": tile_ms / max(tile_n, 1),
                                    "hbm_frac": ((b_cheb if method == N.METHOD_CHEB else b_passb)
                                                 / (tile_ms / 1e3 / tile_n) / 1e9 / peak)
                                    if tile_n else None},
                    "schwarz_stages": {"launches": cpl_n, "avg_ms": cpl_ms / max(cpl_n, 1),
                                       "hbm_frac": (b_couple / (cpl_ms / 1e3 / cpl_n) / 1e9 / peak)
                                       if cpl_n else None},
                    "stencil": {"launches": prof["stencil"][1],
                                "avg_ms": prof["stencil"][0] / max(prof["stencil"][1], 1)},
                    "precondition_start": {"launches": prof["precond"][1],
                                           "avg_ms": prof["precond"][0] / max(prof["precond"][1], 1)}},
        "ensemble_c5": ens,
        "fs_barotropic_loop": fs,
        "config_c1_basin": c1,
        "config_c2_1440x720": c2,
        "config_c4_learned_sequence": c4,
        "reference_solver_call_182x92": ref_call,
        "cpu_baseline": cpu,
        "cpu_baseline_forms": cpu_forms,
        "clocks": clk.summary(),
        "gpu_launches": int(launches_value),
        "gpu_launches_e2e": int(launches_e2e),
        # the north-star comparison, last so that a stored tail of the line keeps it
        "value_arm": {"mean_iterations": float(np.mean([r.iterations for r in reps])),
                      "mean_refinements": float(np.mean([r.refinements for r in reps])),
                      "max_rel_residual": float(max(relres)), "status": sorted(set(status)),
                      "max_rel_err_vs_fp64_gpu": float(max(errs))},
        "linear_mixed": {"value": world * K / t_lin, "unit": "solves/s",
                         "ms_per_step": 1e3 * t_lin / K,
                         "mean_iterations": float(np.mean([r.iterations for r in reps_lin]))},
        "fp64_plain": {"value": world * K / t_fp64, "unit": "solves/s",
                       "ms_per_step": 1e3 * t_fp64 / K,
                       "mean_iterations": float(np.mean(it64)),
                       "preconditioner": "block-Jacobi tiles"},
        "speedup_vs_fp64_plain": (K / t_value) / (K / t_fp64),
        "linear_mixed_speedup_vs_fp64_plain": (K / t_lin) / (K / t_fp64),
        "error_vs_cpu_oracle": oracle_err,
    }
    if rank == 0:
        print(json.dumps(line), flush=True)
    if warm is not None:
        warm.close()
    solver.close()
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


def run_profile(args):
    """A small case for ncu: no timing, no JSON line."""
    import ctypes as C

    import torch

    from musoc_solver_b200 import build, native as N, problems as P
    from musoc_solver_b200.solver import SevpSolver

    build.build()
    if args.profile == "solve":
        p = P.global_grid(args.nx, args.ny, seed=11)
        tiles = (16, 6) if args.tiles == "auto" else tuple(int(v) for v in args.tiles.split("x"))
        s = SevpSolver(p, tile_m=tiles[0], tile_h=tiles[1], growth_limit=GROWTH,
                       schwarz=args.precond == "schwarz")
        s.set_pass_b_kernel(PASS_B_KINDS[args.pass_b])
        b = torch.from_numpy(p.b).cuda()
        if args.method == "cheb":
            s.chebyshev_setup(b)
            s.set_method(N.METHOD_CHEB)
        _, rep = s.solve(b, precision=args.profile_precision, max_iter=args.profile_max_iter)
        torch.cuda.synchronize()
        print("ok", rep)
        s.close()
        return 0
    from musoc_solver_b200.unet import lib as nnlib

    H, W, cin, cout = (int(v) for v in args.conv.split(","))
    L = nnlib()
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(H * W, cin, device="cuda", generator=g).to(torch.bfloat16)
    wk = (torch.randn(9, cout, cin, device="cuda", generator=g) / 30).to(torch.bfloat16)
    bias = torch.zeros(cout, device="cuda")
    y = torch.zeros(H * W, cout, dtype=torch.bfloat16, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    for _ in range(3):
        st = L.sevp_nn_conv3x3_tma(ptr(x), cin, 0, cin, ptr(wk), ptr(bias), ptr(y), cout, 0, cout,
                                   1, H, W, 1, None)
        assert st == 0, st
    code = C.c_int(-1)
    assert L.sevp_nn_tc_status(C.byref(code)) == 0 and code.value == 0
    torch.cuda.synchronize()
    print("ok", args.conv)
    return 0


def main():
    args = parse()
    # the CPU oracle's OpenMP runtime (tile PCG legs) uses every host core;
    # serial legs (REP, BiCGSTAB, the single-thread baseline) say so
    os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count() or 1))
    if args.profile:
        return run_profile(args)
    world, rank, local, dist = dist_setup(args)
    if args.impl == "reference":
        rc = run_reference(args, world, rank)
        if dist is not None:
            dist.destroy_process_group()
        return rc
    return run_native(args, world, rank, local, dist)


if __name__ == "__main__":
    sys.exit(main())
