"""The work that users of this framework have it do, as cases to be timed.

A case names a kind of call and its sizes:

* ``solve``     one elliptic solve through ``SevpSolver.solve`` (device fields)
* ``step``      one time step of a sequence through ``SevpSolver.solve_step``,
                from the linear extrapolation or the learned guess
* ``ensemble``  all members of an ensemble through ``EnsembleSolver.solve``
* ``fs``        one pass of the barotropic correction loop
                (``BarotropicCorrection.run``: land mask, right-hand side,
                solve, correction of every layer)
* ``pcg_call``  the Fortran call ``p_sevp_pcg_`` on host arrays
* ``rep_call``  the Fortran call ``rep1_`` on host arrays
* ``train``     one training step of the warm start's U-Net

An ocean model has one bathymetry and solves on it every step, so a case's
operator is fixed by its sizes, and the seed makes the fields that change from
step to step: right-hand sides, velocities, histories, network inputs.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from musoc_solver_b200 import native as N
from musoc_solver_b200 import problems as P
from musoc_solver_b200.barotropic import BarotropicCorrection
from musoc_solver_b200.ensemble import EnsembleSolver
from musoc_solver_b200.solver import SevpSolver
from musoc_solver_b200.unet import CONVS, HEAD_C, UNet
from musoc_solver_b200.warmstart import LearnedWarmStart

EARTH_R = 6.371e6
LAT_MAX = 78.0
GRAVITY = 9.81


def listed():
    return [
        # the reference's own grid: FS_SOLVER's Krylov call with PREP's planes,
        # host arrays in and out, the operator found again by its hash
        dict(name="pcg_call_180x90", kind="pcg_call", nx=180, ny=90),
        # the same grid's direct solve: REP1 on 15 row blocks, influence data
        # from PRE1, device copies of it kept (sevp_dropin_cache)
        dict(name="rep1_call_180x90", kind="rep_call", nx=180, ny=90, blocks=15),
        # the smallest native solve: closed 96 x 96 basin, FP64, 24 x 24 tiles
        dict(name="basin_96_fp64", kind="solve", grid="basin", nx=96, ny=96, tile_m=24, tile_h=24,
             precision=0, schwarz=False, inner_tol=1e-5),
        # 0.25 degree global grid, plain FP64 PCG
        dict(name="global_1440x720_fp64", kind="solve", grid="global", nx=1440, ny=720, tile_m=16,
             tile_h=6, precision=0, schwarz=False, inner_tol=1e-5),
        # a regional-size odd grid with every default of the Python interface
        # (16 x 16 tiles, ragged in both directions), mixed precision
        dict(name="global_1203x601_mixed", kind="solve", grid="global", nx=1203, ny=601, tile_m=16,
             tile_h=16, precision=1, schwarz=False, inner_tol=1e-5),
        # one step of the 400-step 0.25 degree sequence with the network's guess
        dict(name="step_1440x720_learned", kind="step", nx=1440, ny=720, tile_m=16, tile_h=8,
             guess="learned", coarse=4, inner_tol=1e-5),
        # one step of the 0.1 degree sequence, mixed precision from the linear
        # extrapolation, with the tile shape and tolerance the autotuner picks
        dict(name="step_3600x2400_linear", kind="step", nx=3600, ny=2400, tile_m=16, tile_h=6,
             guess="linear", coarse=0, inner_tol=1e-4),
        # the same grid in plain FP64 from zero
        dict(name="global_3600x2400_fp64", kind="solve", grid="global", nx=3600, ny=2400,
             tile_m=16, tile_h=6, precision=0, schwarz=False, inner_tol=1e-5),
        # the 64-member ensemble in mixed precision
        dict(name="ensemble_64x720x360", kind="ensemble", members=64, nx=720, ny=360, precision=1,
             schwarz=False),
        # a smaller ensemble in FP64 with the overlapping Schwarz preconditioner
        # (the fastest choice for its well-conditioned members)
        dict(name="ensemble_16x720x360_schwarz", kind="ensemble", members=16, nx=720, ny=360,
             precision=0, schwarz=True),
        # one pass of the barotropic correction at 0.5 degree with 20 layers
        dict(name="fs_720x360x20", kind="fs", nx=720, ny=360, layers=20),
        # one training step of the network on the 1/4 grid of 1440 x 720
        dict(name="train_184x360", kind="train", height=184, width=360),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "step", "step", "ensemble", "fs", "pcg_call",
                       "rep_call", "train"])
    if kind == "pcg_call":
        nx = _log(rng, 60, 360)
        return dict(kind=kind, nx=nx, ny=max(24, int(nx * rng.uniform(0.4, 0.6))))
    if kind == "rep_call":
        # row blocks of 6, the last one 5 to 7 rows
        nx = _log(rng, 48, 200)
        blocks = max(4, int(nx * rng.uniform(0.4, 0.6)) // 6)
        return dict(kind=kind, nx=nx, ny=6 * blocks + rng.choice([-1, 0, 1]), blocks=blocks)
    if kind == "train":
        return dict(kind=kind, height=8 * _log(rng, 6, 36), width=8 * _log(rng, 9, 60))
    if kind == "fs":
        nx = _log(rng, 120, 900)
        return dict(kind=kind, nx=nx, ny=int(nx * rng.uniform(0.4, 0.6)),
                    layers=rng.choice([6, 10, 17, 20, 25]))
    if kind == "ensemble":
        schwarz = rng.random() < 0.4
        return dict(kind=kind, members=rng.choice([3, 8, 16, 24, 40]), nx=_log(rng, 90, 720),
                    ny=6 * _log(rng, 8, 60), precision=rng.choice([0, 1]), schwarz=schwarz)
    nx = _log(rng, 90, 2400)
    ny = int(nx * rng.uniform(0.4, 0.67))
    tile_m, tile_h = rng.choice([(16, 16), (16, 6), (16, 6), (16, 8), (8, 8)])
    if kind == "step":
        guess = rng.choice(["linear", "linear", "learned"])
        coarse = 0
        if guess == "learned":
            coarse = rng.choice([4, 8])
            nx, ny = max(240, nx) // coarse * coarse, max(120, ny) // coarse * coarse
        return dict(kind=kind, nx=nx, ny=ny, tile_m=tile_m, tile_h=tile_h, guess=guess,
                    coarse=coarse, inner_tol=rng.choice([1e-4, 1e-5]))
    schwarz = tile_h <= 8 and rng.random() < 0.3
    return dict(kind=kind, grid="global", nx=nx, ny=ny, tile_m=tile_m, tile_h=tile_h,
                precision=rng.choice([0, 1]), schwarz=schwarz, inner_tol=1e-5)


# ------------------------------------------------------------------ grids
@functools.lru_cache(maxsize=2)
def _global(nx, ny):
    return P.global_grid(nx, ny, seed=1)


@functools.lru_cache(maxsize=2)
def _basin(n):
    return P.basin(seed=0, n=n)


@functools.lru_cache(maxsize=2)
def _members(members, nx, ny):
    return P.ensemble(members=members, nx=nx, ny=ny, seed=5)


@functools.lru_cache(maxsize=2)
def _layered(nx, ny, layers):
    return P.fs_state(nx, ny, layers, seed=7)


@functools.lru_cache(maxsize=2)
def _prep(nx, ny):
    return P.prep_grid(nx, ny, seed=0)


@functools.lru_cache(maxsize=2)
def _rep(nx, ny, blocks):
    """The reference's test stencil (AC shifted so that it is not singular),
    its row blocks and PRE1's influence data."""
    p = P.idealised(nx, ny)
    p.ac[:] += np.float32(0.01)
    planes = [np.ascontiguousarray(a, np.float32) for a in p.coeffs()]
    ie = np.zeros(blocks, np.int32)
    N.check(N.lib().sevp_block_partition(ny, blocks, 3, N.ptr(ie)), "sevp_block_partition")
    rinv, rinv1 = np.zeros((blocks, nx, nx)), np.zeros((blocks - 1, nx, nx))
    h = np.zeros((ny + 2, nx + 2))
    N.lib().sevp_set_periodic_we(1)
    N.lib().pre1_(*[N.ptr(a) for a in planes], N.ptr(rinv), N.ptr(rinv1), N.ptr(h), N.ptr(ie),
                  N.iref(nx + 2), N.iref(nx), N.iref(blocks))
    N.check(N.lib().sevp_last_status(), "pre1_")
    return p, planes, ie, rinv, rinv1


# ----------------------------------------------------------------- fields
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _smooth(shape, scale, g):
    """Unit-variance random fields with Gaussian spectral falloff, periodic
    in the last two axes; scale is the correlation length in cells."""
    w = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.rfft2(w)
    ky = torch.fft.fftfreq(shape[-2], device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(shape[-1], device="cuda", dtype=torch.float64)[None, :]
    f *= torch.exp(-((kx**2 + ky**2) * (math.pi * scale) ** 2))
    out = torch.fft.irfft2(f, s=shape[-2:])
    out -= out.mean(dim=(-2, -1), keepdim=True)
    return out / out.std(dim=(-2, -1), keepdim=True)


def _divergence(depth, g):
    """Volume-flux divergence of smooth random velocities through the wet
    faces of global grids, depth (..., ny, nx) on the device."""
    ny, nx = depth.shape[-2:]
    dy = EARTH_R * math.radians(2 * LAT_MAX / ny)
    lat_f = torch.arange(1, ny, device="cuda", dtype=torch.float64) * (2 * LAT_MAX / ny) - LAT_MAX
    dxf = EARTH_R * math.radians(360.0 / nx) * torch.cos(torch.deg2rad(lat_f))
    scale = max(nx / 60.0, 2.0)
    u, v = 0.1 * _smooth(depth.shape, scale, g), 0.1 * _smooth(depth.shape, scale, g)
    wet, east = depth > 0, torch.roll(depth, -1, -1)
    fx = torch.where(wet & (east > 0), 0.5 * (depth + east) * u * dy, 0.0)
    south, north = depth[..., :-1, :], depth[..., 1:, :]
    fy = torch.where((south > 0) & (north > 0),
                     0.5 * (south + north) * v[..., :-1, :] * dxf[:, None], 0.0)
    div = fx - torch.roll(fx, 1, -1)
    div[..., :-1, :] += fy
    div[..., 1:, :] -= fy
    return div


def _solve_rhs(case, seed):
    if case["grid"] == "basin":
        p = _basin(case["nx"])
        noise = torch.randn((p.ny, p.nx), generator=_gen(seed), device="cuda", dtype=torch.float64)
        return p, 1e-6 * noise * torch.from_numpy(p.meta["wet"] * p.meta["area"]).cuda()
    p = _global(case["nx"], case["ny"])
    return p, _divergence(torch.from_numpy(p.meta["depth"]).cuda(), _gen(seed))


def _step_rhs(case, seed):
    """Right-hand sides of three successive steps of an eddy sequence."""
    p = _global(case["nx"], case["ny"])
    wet = torch.from_numpy(p.meta["wet"]).cuda()
    seq = P.eddy_rhs(case["nx"], case["ny"], range(40, 43), seed=int(seed) + 100)
    return p, [torch.where(wet, torch.from_numpy(b).cuda(), 0.0) for _, b in seq]


def _ensemble_rhs(case, seed):
    ms = _members(case["members"], case["nx"], case["ny"])
    depth = torch.from_numpy(np.stack([m.meta["depth"] for m in ms])).cuda()
    return ms, _divergence(depth, _gen(seed)).reshape(-1, case["nx"])


def _velocities(case, seed):
    """White-noise layer velocities (0.1 m/s), as the loop's own test state has."""
    i0, j0, k1 = case["nx"] + 2, case["ny"] + 2, case["layers"]
    g = _gen(seed)
    u = 0.1 * torch.randn((k1, j0, i0), generator=g, device="cuda")
    return u, 0.1 * torch.randn((k1, j0 - 1, i0), generator=g, device="cuda")


def _call_rhs(case, seed):
    """REAL*4 noise right-hand side of a Fortran call (host)."""
    f = np.random.default_rng(int(seed)).standard_normal((case["ny"], case["nx"]))
    if case["kind"] == "pcg_call":
        f *= float(np.abs(_prep(case["nx"], case["ny"]).ac).mean())
    return f.astype(np.float32)


def _network(case, seed):
    """Weights of a He-initialised network (FP32), its normalised inputs (the
    first three of 16 channels) and the target on the network grid."""
    g = _gen(seed)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    st = {}
    for name, ci, co in CONVS:
        w = r(9, ci, co) * math.sqrt(2.0 / (9 * (3 if name == "enc0a" else ci)))
        if name == "enc0a":
            w[:, 3:] = 0.0
        st[name + ".0"], st[name + ".1"] = w, 0.02 * r(co)
    st["head.0"], st["head.1"] = 0.1 * r(HEAD_C), 0.02 * r(1)
    h, w = case["height"], case["width"]
    f = _smooth((4, h, w), 4.0, g)
    x = torch.zeros((h * w, 16), device="cuda", dtype=torch.bfloat16)
    x[:, :3] = f[:3].reshape(3, -1).t().to(torch.bfloat16)
    return st, x, f[3].reshape(-1).float().contiguous()


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_solve(case, seed):
    p, b = _solve_rhs(case, seed)
    s = SevpSolver(p, tile_m=case["tile_m"], tile_h=case["tile_h"], schwarz=case["schwarz"])
    return dict(case=case, s=s, b=b, x=torch.zeros_like(b))


def _prepare_step(case, seed):
    p, (b0, b1, b2) = _step_rhs(case, seed)
    s = SevpSolver(p, tile_m=case["tile_m"], tile_h=case["tile_h"])
    eta2 = s.solve(b0)[0]
    eta1 = s.solve(b1, x=eta2.clone())[0]
    warm = None
    if case["guess"] == "learned":
        warm = LearnedWarmStart.create(s, train=False, coarse=case["coarse"])
        warm.attach()
    return dict(case=case, s=s, b=b2, eta1=eta1, eta2=eta2, x=torch.zeros_like(b2), warm=warm)


def _prepare_ensemble(case, seed):
    ms, b = _ensemble_rhs(case, seed)
    e = EnsembleSolver(ms, schwarz=case["schwarz"])
    return dict(case=case, e=e, b=b, x=torch.zeros_like(b), tol=e.stacked_tol(b))


def _prepare_fs(case, seed):
    st = _layered(case["nx"], case["ny"], case["layers"])
    u0, v0 = _velocities(case, seed)
    p0 = torch.zeros((case["ny"] + 2, case["nx"] + 2), device="cuda")
    scr = torch.zeros((4, case["ny"] + 2, case["nx"] + 2), device="cuda")
    return dict(case=case, bc=BarotropicCorrection(st), u0=u0, v0=v0, u=u0.clone(), v=v0.clone(),
                p0=p0, scr=scr)


def _prepare_pcg_call(case, seed):
    p = _prep(case["nx"], case["ny"])
    N.lib().sevp_set_periodic_we(1)
    return dict(case=case, planes=p.coeffs(), f=_call_rhs(case, seed),
                x=np.zeros((case["ny"] + 2, case["nx"] + 2)))


def _prepare_rep_call(case, seed):
    nx, ny, nb = case["nx"], case["ny"], case["blocks"]
    _, planes, ie, rinv, rinv1 = _rep(nx, ny, nb)
    N.lib().sevp_set_periodic_we(1)
    N.check(N.lib().sevp_dropin_cache(1), "sevp_dropin_cache")
    return dict(case=case, planes=planes, ie=ie, rinv=rinv, rinv1=rinv1, f=_call_rhs(case, seed),
                d0=np.zeros((nb - 1, nx)), d1=np.zeros(nx), d2=np.zeros(nx),
                h=np.zeros((ny + 2, nx + 2)), x=np.zeros((ny + 2, nx + 2)))


def _prepare_train(case, seed):
    st, x, t = _network(case, seed)
    net = UNet(case["height"], case["width"])
    net.load_state({k: v.cpu().numpy() for k, v in st.items()})
    net.A["x"].copy_(x)
    return dict(case=case, net=net, t=t)


# -------------------------------------------------------------------- run
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state, state["case"])


def _run_solve(s, case):
    return s["s"].solve(s["b"], x=s["x"], x_is_guess=False, precision=case["precision"],
                        inner_tol=case["inner_tol"])[0]


def _run_step(s, case):
    guess = N.GUESS_LEARNED if case["guess"] == "learned" else N.GUESS_LINEAR
    return s["s"].solve_step(s["b"], s["eta1"], s["eta2"], s["x"], guess=guess, precision=1,
                             inner_tol=case["inner_tol"])[0]


def _run_ensemble(s, case):
    return s["e"].solve(s["b"], x=s["x"], precision=case["precision"], residuals=False,
                        tol_stack=s["tol"], x_is_guess=False)[0]


def _run_fs(s, case):
    # the momentum step's new velocities, then the correction of this step
    s["u"].copy_(s["u0"])
    s["v"].copy_(s["v0"])
    s["p0"].zero_()
    s["scr"].zero_()
    s["bc"].run(s["u"], s["v"], s["p0"], s["scr"], tolerance=0.0, mxmask=1)
    return [s["u"], s["v"], s["p0"], s["scr"]]


def _run_pcg_call(s, case):
    planes = [N.ptr(a) for a in s["planes"]]
    s["x"].fill(0.0)
    N.lib().p_sevp_pcg_(*planes, N.ptr(s["f"]), N.ptr(s["x"]), *planes, N.iref(case["nx"]),
                        N.iref(case["ny"]))
    N.check(N.lib().sevp_last_status(), "p_sevp_pcg_")
    return s["x"]


def _run_rep_call(s, case):
    s["x"].fill(0.0)
    N.lib().rep1_(*[N.ptr(a) for a in s["planes"]], N.ptr(s["rinv"]), N.ptr(s["rinv1"]),
                  N.ptr(s["d0"]), N.ptr(s["d1"]), N.ptr(s["d2"]), N.ptr(s["f"]), N.ptr(s["h"]),
                  N.ptr(s["x"]), N.ptr(s["ie"]), N.iref(case["nx"] + 2), N.iref(case["nx"]),
                  N.iref(case["blocks"]))
    N.check(N.lib().sevp_last_status(), "rep1_")
    return s["x"]


def _run_train(s, case):
    net = s["net"]
    y = net.forward()
    net.backward(s["t"])
    net.adam_step(lr=1e-3)
    return dict(y=y, loss=net.loss, grads={n: list(g) for n, g in net.gw.items()})


# ------------------------------------------------------------------- work
def work(case):
    """One read of every input and one write of every output; the flops of
    two applications of the operator (a solve cannot do without forming a
    residual and checking it), or of the network's convolutions."""
    kind = case["kind"]
    if kind == "train":
        p = case["height"] * case["width"]
        at = lambda name: 4 ** {"0": 0, "1": 1, "2": 2}.get(name.rstrip("ab")[-1:], 3)  # noqa: E731
        fl = sum(18.0 * ci * co * p / at(n) * (2 if n == "enc0a" else 3) for n, ci, co in CONVS)
        weights = sum(9 * ci * co for _, ci, co in CONVS)
        return dict(bytes=32.0 * p + 8 * p + 32.0 * weights, flops=fl)
    n = float(case["nx"] * case["ny"] * case.get("members", 1))
    if kind == "rep_call":
        influence = 8.0 * case["nx"] ** 2 * (2 * case["blocks"] - 1)
        return dict(bytes=n * 32 + influence, flops=influence / 2)
    if kind == "fs":
        return dict(bytes=n * (12 + 20 * case["layers"] + 24), flops=n * (18 + 12 * case["layers"]))
    return dict(bytes=n * (28 + (16 if kind == "step" else 0)), flops=18.0 * n)


# ------------------------------------------------------------------ exact
def _planes64(p):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda().double() for a in p.coeffs()]


def _apply(c, x, periodic):
    al, ab, ac, ar, at = c
    y = ac * x
    y[1:] += ab[1:] * x[:-1]
    y[:-1] += at[:-1] * x[1:]
    if periodic:
        y += al * torch.roll(x, 1, 1) + ar * torch.roll(x, -1, 1)
    else:
        y[:, 1:] += al[:, 1:] * x[:, :-1]
        y[:, :-1] += ar[:, :-1] * x[:, 1:]
    return y


def _symmetric(c, periodic):
    """The planes with each coupling the mean of its two sides."""
    al, ab, ac, ar, at = [a.clone() for a in c]
    ab[0], at[-1] = 0.0, 0.0
    ab[1:] = at[:-1] = 0.5 * (ab[1:] + at[:-1])
    ar = 0.5 * (ar + torch.roll(al, -1, 1))
    if not periodic:
        ar[:, -1] = 0.0
    return torch.roll(ar, 1, 1), ab, ac, ar, at


def _solve64(c, b, periodic, w=None, rounds=3):
    """A x = b in FP64: Jacobi-preconditioned CG on the row-scaled symmetric
    part, repeated on the residual of A itself."""
    w = torch.ones((b.shape[0], 1), dtype=torch.float64, device="cuda") if w is None else w
    sym = _symmetric([w * a for a in c], periodic)
    x = torch.zeros_like(b)
    for _ in range(rounds):
        r = w * (b - _apply(c, x, periodic))
        d = torch.zeros_like(b)
        z = r / sym[2]
        p, rz, r0 = z.clone(), (r * z).sum(), float(r.norm())
        for k in range(20000):
            q = _apply(sym, p, periodic)
            a = rz / (p * q).sum()
            d += a * p
            r -= a * q
            if k % 20 == 19 and float(r.norm()) <= 1e-9 * r0:
                break
            z = r / sym[2]
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        x += d
    return x


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _exact_solve(case, seed):
    p, b = _solve_rhs(case, seed)
    return _solve64(_planes64(p), b, p.periodic)


def _exact_step(case, seed):
    p, rhs = _step_rhs(case, seed)
    return _solve64(_planes64(p), rhs[2], p.periodic)


def _exact_ensemble(case, seed):
    ms, b = _ensemble_rhs(case, seed)
    c = [torch.cat(k) for k in zip(*[_planes64(m) for m in ms])]
    return _solve64(c, b, True)


def _exact_pcg_call(case, seed):
    p = _prep(case["nx"], case["ny"])
    w = 1.0 / (p.meta["ocs"][1:-1].astype(np.float64) * p.meta["ody"][1:-1])
    f = torch.from_numpy(_call_rhs(case, seed)).cuda().double()
    return _ghosted(_solve64(_planes64(p), f, True, torch.from_numpy(w).cuda()[:, None]))


def _exact_rep_call(case, seed):
    p = P.idealised(case["nx"], case["ny"])
    p.ac[:] += np.float32(0.01)
    f = torch.from_numpy(_call_rhs(case, seed)).cuda().double()
    return _ghosted(_solve64(_planes64(p), f, True))


def _ghosted(x):
    """The padded field of a Fortran call: zero ghost rows, periodic columns."""
    out = np.zeros((x.shape[0] + 2, x.shape[1] + 2))
    out[1:-1, 1:-1] = x.cpu().numpy()
    out[1:-1, 0], out[1:-1, -1] = out[1:-1, -2], out[1:-1, 1]
    return out


def _exact_fs(case, seed):
    st = _layered(case["nx"], case["ny"], case["layers"])
    d = {k: torch.from_numpy(np.ascontiguousarray(getattr(st, k))).cuda().double()
         for k in ("iu0", "iv0", "iu", "iv", "odx", "ody", "ocs", "csv", "odyv", "odz", "rscale")}
    u, v = (t.double() for t in _velocities(case, seed))
    u[0, 1:-1, 1:-2] *= d["iu0"][1:-1, 1:-2]
    u[0, 1:-1, 0] *= d["iu0"][1:-1, 0]
    u[0, 1:-1, -2] *= d["iu0"][1:-1, -2]
    v[0, 1:-1, 1:-1] *= d["iv0"][1:-2, 1:-1]
    col = lambda a: a[:, None]  # noqa: E731
    s = torch.zeros_like(u[0, 1:-1, 1:-1])
    for k in range(case["layers"]):
        fx = (u[k, 1:-1, 1:-1] - u[k, 1:-1, :-2]) * col(d["odx"][1:-1])
        fy = col(d["csv"][1:]) * v[k, 1:, 1:-1] - col(d["csv"][:-1]) * v[k, :-1, 1:-1]
        s += (fx + fy * col(d["ocs"][1:-1] * d["ody"][1:-1])) / d["odz"][k]
    x = _solve64(_planes64(st.problem), s * col(d["rscale"]), True)
    p0 = torch.zeros_like(u[0])
    p0[1:-1, 1:-1] = float(st.odt) * x
    scr = torch.zeros((4, *u[0].shape), dtype=torch.float64, device="cuda")
    cu = -(torch.roll(x, -1, 1) - x) * col(d["odx"][1:-1])
    scr[0, 1:-1, 1:-1] = cu
    scr[0, 1:-1, 0] = cu[:, -1]
    scr[1, 1:-2, 1:-1] = -(x[1:] - x[:-1]) * col(d["odyv"][1:-1])
    scr[2:] = scr[:2]
    u[0] += scr[0]
    v[0] += scr[1, :-1]
    u[1:] += scr[0] * d["iu"][1:]
    v[1:] += scr[1, :-1] * d["iv"][1:]
    return [u, v, p0, scr]


def _exact_train(case, seed):
    st, x, t = _network(case, seed)
    h, w = case["height"], case["width"]
    par = {k: (a.to(torch.bfloat16) if a.dim() == 3 else a).double().requires_grad_(True)
           for k, a in st.items()}
    f = torch.nn.functional

    def conv(name, a):
        k = par[name + ".0"].reshape(3, 3, *par[name + ".0"].shape[1:]).permute(3, 2, 0, 1)
        return f.relu(f.conv2d(a, k, par[name + ".1"], padding=1))

    pool = lambda a: f.avg_pool2d(a, 2)  # noqa: E731
    up = lambda a: f.interpolate(a, scale_factor=2, mode="nearest")  # noqa: E731
    e0 = conv("enc0b", conv("enc0a", x.double().t().reshape(1, 16, h, w)))
    e1 = conv("enc1b", conv("enc1a", pool(e0)))
    e2 = conv("enc2b", conv("enc2a", pool(e1)))
    a = conv("botb", conv("bota", pool(e2)))
    for lvl, skip in ((2, e2), (1, e1), (0, e0)):
        a = torch.cat([conv("up%d" % lvl, up(a)), skip], 1)
        a = conv("dec%db" % lvl, conv("dec%da" % lvl, a))
    y = (a * par["head.0"].reshape(1, -1, 1, 1)).sum(1).reshape(-1) + par["head.1"]
    loss = ((y - t.double()) ** 2).mean()
    loss.backward()
    names = [n for n, _, _ in CONVS] + ["head"]
    grads = {n: [par[n + ".0"].grad, par[n + ".1"].grad] for n in names}
    grads["enc0a"][0][:, 3:] = 0.0
    return dict(y=y.detach(), loss=loss.detach().reshape(1), grads=grads)
