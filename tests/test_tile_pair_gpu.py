"""The two-column tile pass (SEVP_PASS_B_PAIRS) at the sizes where its mapping
can go wrong: every lane-segment width (8, 16, 32 columns) full and narrower,
odd tile widths and odd grids (no vector copies), narrow last tiles and short
last tile rows, tile heights below, at, between and above the register heights
(6 and 8), sub-block counts that differ between the two halves of a warp, one
tile per grid, and caller buffers that are aligned to one value only.

z = M^-1 r against the CPU oracle's tile solve.  Tolerances, of max|z|: 1e-8
in FP64 (the marching amplifies rounding by at most the growth bound 1e6 on
top of ~1e-16; the two march in different orders), 1e-6 in FP32 vectors (r and
z rounded to FP32, 6e-8 each, times the tile operator's condition, at most
about 10 on these grids).
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


# (nx, ny, tile columns, tile rows, growth limit)
CASES = [
    (128, 66, 16, 6, 1e6),    # vector and 16-byte copies, full tiles
    (130, 64, 16, 6, 1e6),    # nx even, not a multiple of 4
    (131, 65, 16, 6, 1e6),    # odd grid, ragged both ways
    (96, 48, 8, 8, 1e6),
    (100, 50, 8, 6, 1e3),
    (224, 64, 32, 8, 1e6),
    (150, 77, 24, 7, 1e4),    # 24 of 32 lanes' columns, rows between 6 and 8
    (90, 45, 5, 4, 1e6),      # odd tile width
    (120, 60, 12, 6, 1e2),    # many sub-blocks
    (33, 17, 16, 6, 1e3),
    (7, 3, 8, 6, 1e6),        # one partial tile
    (128, 64, 16, 16, 1e6),   # rows staged in shared memory
    (131, 65, 16, 9, 1e3),
    (96, 96, 24, 24, 1e6),
    (150, 70, 32, 32, 1e4),
]


@pytest.mark.parametrize("nx,ny,tm,th,growth", CASES)
@pytest.mark.parametrize("offset", [0, 1])
def test_tile_pair_matches_oracle(torch_cuda, oracle, nx, ny, tm, th, growth, offset):
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_cuda
    p = P.basin(2, n=7) if nx == 7 else P.global_grid(nx, ny, seed=3)
    nx, ny = p.nx, p.ny
    s = SevpSolver(p, tile_m=tm, tile_h=th, growth_limit=growth)
    pc = oracle.TilePC(p, tm, th, tile_nb=s.tile_nb)
    r = np.random.default_rng(4).standard_normal((ny, nx))
    zo = pc.apply(r)
    scale = np.abs(zo).max()
    for dt, tol in ((torch.float64, 1e-8), (torch.float32, 1e-6)):
        # offset 1: the buffer starts one value past an aligned address
        buf = torch.zeros(nx * ny + 1, dtype=dt, device="cuda")
        rd = buf[offset:offset + nx * ny].reshape(ny, nx)
        rd.copy_(torch.from_numpy(r))
        z = s.precondition(rd).double().cpu().numpy()
        assert np.abs(z - zo).max() <= tol * scale, (dt, np.abs(z - zo).max() / scale)
    s.close()
