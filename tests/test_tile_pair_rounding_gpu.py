"""The two-column tile pass in FP64: every marched row is the rounded quotient.

A tile's rows come from z_{k+1} = q_k / AT_k, with q_k = r_k less the terms of
the rows below, one fused multiply-add each (south, the lane's other column,
centre, then the neighbour lane's column).  With one sub-block per tile the
rows that the pass returns are the ones it marched, so from them each q_k is
reproduced exactly in rational arithmetic, and z_{k+1} must equal q_k / AT_k
rounded once: bit for bit, no tolerance.  Full tiles in registers (16 x 6, 8 x
8, 32 x 6), the rolled loops (16 x 4, 24 x 24, odd tile and grid widths).
"""
from fractions import Fraction

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


def _fma(c, v, p):
    """p - c v, rounded once."""
    return float(Fraction(p) - Fraction(c) * Fraction(v))


# (nx, ny, tile columns, tile rows)
CASES = [(64, 24, 16, 6), (66, 26, 8, 8), (64, 18, 32, 6), (48, 16, 16, 4), (48, 24, 24, 24),
         (45, 21, 19, 7), (33, 32, 16, 16)]


@pytest.mark.parametrize("nx,ny,tm,th", CASES)
def test_marched_rows_are_rounded_quotients(torch_cuda, nx, ny, tm, th):
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_cuda
    p = P.global_grid(nx, ny, seed=3)
    s = SevpSolver(p, tile_m=tm, tile_h=th, sub_rows=th)
    r = np.random.default_rng(5).standard_normal((ny, nx))
    z = s.precondition(torch.from_numpy(r).cuda()).cpu().numpy()
    _, _, ac, ar, at = (a.astype(np.float64) for a in p.coeffs())
    assert np.max(s.tile_nb) == 1
    for b, a in np.ndindex(-(-ny // th), -(-nx // tm)):
        j0, i0 = b * th, a * tm
        hh, mw = min(th, ny - j0), min(tm, nx - i0)
        for k in range(hh - 1):
            j = j0 + k
            for n in range(mw):
                i = i0 + n
                q = float(r[j, i])
                if k > 0:
                    q = _fma(at[j - 1, i], z[j - 1, i], q)
                east = (ar[j, i], z[j, i + 1]) if n + 1 < mw else (0.0, 0.0)
                west = (ar[j, i - 1], z[j, i - 1]) if n > 0 else (0.0, 0.0)
                lane, other = (east, west) if n % 2 == 0 else (west, east)
                for c, v in (lane, (ac[j, i], z[j, i]), other):
                    q = _fma(c, v, q)
                want = float(Fraction(q) / Fraction(float(at[j, i])))
                assert z[j + 1, i] == want, (b, a, k, n, z[j + 1, i], want)
    s.close()
