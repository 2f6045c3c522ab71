"""The iterate after a given number of PCG iterations, against the CPU oracle's.

Pass A adds the step of the iteration before it to x, and what ends a run adds
the last one (a kernel of its own in FP64, the residual pass in mixed solves).
A lost or doubled step would only slow the convergence of a whole solve, so
here the iteration cap ends the run after 1 to 6 iterations (odd and even: the
direction buffers alternate; one iteration: x is written once) and x is
compared point by point.  Tolerances, of max|x|: FP64 1e-9 (growth limit 1e4:
the tile solves agree to about 1e-12, and six steps amplify that by less than
a thousand), mixed 1e-5 (FP32 runs: 6e-8 per operation, by less than a
hundred).  The oracle's own iterates k and k - 1 must lie further apart than
forty tolerances (a time step of 300 s: 16 iterations to 1e-12), so that a
wrong step cannot pass.
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


# (nx, ny, tile columns, tile rows): tensor-copied and column-walking pass A
CASES = [(128, 66, 16, 6), (131, 65, 16, 6), (120, 60, 12, 6), (128, 64, 16, 16)]


@pytest.mark.parametrize("nx,ny,tm,th", CASES)
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kernel", [0, 2])  # one-column and two-column tile pass
def test_iterate_after_k_iterations(torch_cuda, oracle, nx, ny, tm, th, precision, kernel):
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_cuda
    p = P.global_grid(nx, ny, seed=3, dt=300.0)
    s = SevpSolver(p, tile_m=tm, tile_h=th, growth_limit=1e4)
    s.set_pass_b_kernel(kernel)
    pc = oracle.TilePC(p, tm, th, tile_nb=s.tile_nb)
    b = torch.from_numpy(p.b).cuda()
    tol = 1e-9 if precision == 0 else 1e-5
    guess = np.random.default_rng(6).standard_normal(p.b.shape) * np.abs(pc.pcg(p.b)[0]).max()
    for x0 in (None, guess):
        before = np.zeros_like(p.b) if x0 is None else x0
        for k in range(1, 7):
            xo, it, _ = pc.pcg(p.b, x0=x0, tol=1e-300, maxit=k)
            assert it == k
            scale = np.abs(xo).max()
            assert np.abs(xo - before).max() > 40 * tol * scale, k
            before = xo
            for check_every in (1, 4):
                xg = None if x0 is None else torch.from_numpy(x0.copy()).cuda()
                x, rep = s.solve(b, xg, precision=precision, tol=1e-300, inner_tol=1e-30,
                                 max_iter=k, check_every=check_every)
                assert rep.iterations == k and rep.status != 0, rep
                err = np.abs(x.cpu().numpy() - xo).max() / scale
                assert err <= tol, (k, check_every, err)
    s.close()
