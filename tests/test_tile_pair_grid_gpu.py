"""The two-column tile pass launches a warp for every task while they all fit.

Tall tiles take so much shared memory per warp that the number of resident
CTAs depends on the CTA's size; the grid must be bounded by the number that
belongs to the size launched.  The launch's grid and block are read from the
profiler's record of sevp_precondition: with at most two tasks per SM and
room for two warps per SM at every shape here (at most 100 KB per warp), the
warps must be at least as many as the tasks, so that none waits for another.
"""
import json

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


@pytest.mark.parametrize("nx,ny,tm,th", [(592, 344, 16, 16), (704, 360, 16, 16), (896, 448, 32, 24),
                                         (600, 300, 24, 16), (180, 90, 16, 16)])
@pytest.mark.parametrize("fp32", [False, True])
def test_every_task_has_a_warp(torch_cuda, tmp_path, nx, ny, tm, th, fp32):
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_cuda
    s = SevpSolver(P.global_grid(nx, ny, seed=1), tile_m=tm, tile_h=th)
    r = torch.ones((ny, nx), dtype=torch.float32 if fp32 else torch.float64, device="cuda")
    s.precondition(r)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        s.precondition(r)
        torch.cuda.synchronize()
    path = tmp_path / "trace.json"
    prof.export_chrome_trace(str(path))
    ev = [e for e in json.loads(path.read_text())["traceEvents"]
          if "k_tile_pair" in e.get("name", "") and "grid" in e.get("args", {})]
    assert len(ev) == 1, [e.get("name") for e in ev]
    per_warp = 32 // (16 if tm <= 16 else 32)  # tiles of a warp group
    groups = -(-(-(-nx // tm)) // per_warp)
    tasks = -(-ny // th) * (-(-groups // 2))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert tasks <= 2 * sms
    a = ev[0]["args"]
    warps = a["grid"][0] * a["block"][0] // 32
    assert warps >= tasks, (a["grid"], a["block"], tasks)
    s.close()
