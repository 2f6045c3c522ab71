"""A Schwarz solve that is over before it starts does no preconditioner work.

The start pass of a run is queued behind the residual pass, so a solve whose
guess meets the tolerance launches it all the same; every tile pass of it must
then return at once.  The time of the first stage's launch (class 'precond' of
the per-kernel times) in such a solve against that of the same stage when it
works (sevp_precondition): at 2880 x 1440 it works for 50 us and more, a launch
that returns takes a few us with the events around it, so below half is asked.
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


@pytest.mark.parametrize("kernel", [0, 2])  # one-column and two-column tile pass
@pytest.mark.parametrize("precision", [0, 1])
def test_finished_schwarz_solve_skips_its_first_stage(torch_cuda, precision, kernel):
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_cuda
    p = P.global_grid(2880, 1440, seed=2)
    s = SevpSolver(p, tile_m=16, tile_h=6, schwarz=True)
    s.set_pass_b_kernel(kernel)
    b = torch.from_numpy(p.b).cuda()
    x, rep = s.solve(b, precision=precision, tol=1e-10)
    assert rep.status == 0 and rep.iterations > 0
    r = torch.from_numpy(np.random.default_rng(1).standard_normal(p.b.shape)).cuda()
    if precision == 1:
        r = r.float()

    def first_stage(call):
        times = []
        for _ in range(5):
            s.profile(True)
            call()
            ms, n = s.profile_read()["precond"]
            assert n == 1, n
            times.append(ms)
        s.profile(False)
        return float(np.median(times))

    def finished():
        y, again = s.solve(b, x.clone(), precision=precision, tol=1e-8)
        assert again.status == 0 and again.iterations == 0 and torch.equal(y, x)

    works = first_stage(lambda: s.precondition(r))
    over = first_stage(finished)
    assert over < 0.5 * works, (over, works)
    s.close()
