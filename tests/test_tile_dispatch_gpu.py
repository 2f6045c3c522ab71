"""Which tile pass a tiling runs: the two-column pass while all its tasks are
resident or both passes take several rounds, the one-column pass where only the
two-column pass needs a second round and its tiles are small, at heights whose
rows it does not keep in registers, and at widths below the lane segment.

Task counts (two-column) against resident warps, 148 SMs: 16 x 16 tiles 220 of
592 (592 x 344), 1035 of 740 FP64 and 888 FP32 (1440 x 720); 20 x 4 at 592 x 344
1290 of 1036 FP64, 1184 FP32 where the one-column pass's 2580 take two rounds
too.  z is the same operator's either way, to the marching's rounding (1e-8 of
max|z| in FP64 at growth 1e6, as in test_tile_pair_gpu).
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


# (nx, ny, tile columns, tile rows, two-column pass in FP64, in FP32)
CASES = [
    (592, 344, 16, 6, True, True),
    (592, 344, 16, 16, True, True),
    (1440, 720, 16, 16, False, False),
    (720, 360, 16, 1, False, False),
    (2400, 1500, 16, 2, False, True),
    (720, 360, 16, 10, False, False),
    (720, 360, 12, 6, False, False),
    (592, 344, 20, 4, False, True),
    (592, 344, 32, 8, True, True),
    (1203, 601, 17, 12, False, False),
    (1440, 720, 24, 24, True, True),
]


@pytest.mark.parametrize("nx,ny,tm,th,pair64,pair32", CASES)
def test_tile_pass_choice(torch_cuda, nx, ny, tm, th, pair64, pair32):
    from musoc_solver_b200 import native as N
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_cuda
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("task counts are for 148 SMs")
    p = P.global_grid(nx, ny, seed=1)
    s = SevpSolver(p, tile_m=tm, tile_h=th, growth_limit=1e6)
    r = torch.from_numpy(np.random.default_rng(2).standard_normal((ny, nx))).cuda()
    z = s.precondition(r)
    assert s.tile_kernel_used() == (N.PASS_B_PAIRS if pair64 else N.PASS_B_REGISTERS)
    s.solve(torch.from_numpy(p.b).cuda(), precision=1, max_iter=4)
    want = N.PASS_B_PAIRS if pair32 else N.PASS_B_REGISTERS
    assert s.tile_kernel_used() == want and s.pass_b_kernel_used() == want
    s.set_pass_b_kernel(N.PASS_B_REGISTERS)
    z1 = s.precondition(r)
    assert s.tile_kernel_used() == N.PASS_B_REGISTERS
    assert (z - z1).abs().max() <= 1e-8 * z1.abs().max()
    s.close()
