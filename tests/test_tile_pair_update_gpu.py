"""The two-column tile pass as PCG runs it: r -= alpha q, z = M^-1 r, r.z and r.r.

Tilings that reach the kernel (asserted) where its mapping can go wrong: odd
tile widths (17 and 25 columns: value copies, 8-byte matrix copies), 32-lane
segments with 9 and 12 rows, odd and even grids, low growth limits with
different sub-block counts in the two halves of a warp (asserted where named),
and a residual that starts one value past an aligned address.

Bounds: the updated r against numpy's two roundings, two units in the last place
of |r| + |alpha q|; z of that r against the CPU oracle's tile solve, 1e-8 of
max|z| in FP64 and 1e-6 in FP32 (as in test_tile_pair_gpu: growth at most 1e6);
the sums against those of the returned r and z in extended precision, 5e-12 of
the sum of absolute products (at most 22400 terms at 2.2e-16 each).
"""
import numpy as np
import pytest

from musoc_solver_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from musoc_solver_b200 import build

    build.build()
    return torch


# (nx, ny, tile columns, tile rows, growth limit, halves of a warp differ)
CASES = [
    (136, 64, 17, 6, 1e6, True),
    (153, 66, 17, 8, 1e6, True),
    (175, 70, 25, 7, 1e4, False),
    (160, 63, 32, 9, 1e6, True),
    (224, 100, 32, 12, 1e6, True),
    (128, 66, 16, 6, 1e6, True),
    (131, 65, 16, 6, 1e6, True),
    (128, 64, 16, 16, 1e3, False),
    (100, 50, 8, 6, 1e2, False),
]


@pytest.mark.parametrize("nx,ny,tm,th,growth,differ", CASES)
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("fp32", [False, True])
def test_update_pass(torch_cuda, oracle, nx, ny, tm, th, growth, differ, offset, fp32):
    from musoc_solver_b200 import native as N
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_cuda
    p = P.global_grid(nx, ny, seed=3)
    s = SevpSolver(p, tile_m=tm, tile_h=th, growth_limit=growth)
    if differ:
        per = 32 // (8 if tm <= 8 else (16 if tm <= 16 else 32))
        groups = np.asarray(s.tile_nb).reshape(-(-ny // th), -(-nx // tm))[:, ::per]
        pairs = groups.shape[1] // 2 * 2
        assert (groups[:, 0:pairs:2] != groups[:, 1:pairs:2]).any()
    pc = oracle.TilePC(p, tm, th, tile_nb=s.tile_nb)
    dt, npt = (torch.float32, np.float32) if fp32 else (torch.float64, np.float64)
    rng = np.random.default_rng(8)
    r0, q = (rng.standard_normal((ny, nx)).astype(npt) for _ in range(2))
    alpha = 0.375
    buf = torch.zeros(nx * ny + 1, dtype=dt, device="cuda")
    r = buf[offset:offset + nx * ny].reshape(ny, nx)
    r.copy_(torch.from_numpy(r0))
    z, rz, rr = s.pass_b(alpha, r, torch.from_numpy(q).cuda())
    assert s.tile_kernel_used() == N.PASS_B_PAIRS
    r1, z1 = r.cpu().numpy(), z.cpu().numpy()
    ulp = np.finfo(npt).eps
    assert (np.abs(r1 - (r0 - npt(alpha) * q)) <= 2 * ulp * (np.abs(r0) + alpha * np.abs(q))).all()
    zo = pc.apply(r1.astype(np.float64))
    assert np.abs(z1 - zo).max() <= (1e-6 if fp32 else 1e-8) * np.abs(zo).max()
    rl, zl = r1.astype(np.longdouble), z1.astype(np.longdouble)
    assert abs(rz - (rl * zl).sum()) <= 5e-12 * np.abs(rl * zl).sum()
    assert abs(rr - (rl * rl).sum()) <= 5e-12 * (rl * rl).sum()
    s.close()
