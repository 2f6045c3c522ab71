"""Kernels that opt in to large shared memory, on a second device of one process.

The opt-in belongs to the device, so a call on another device after a first one
must make it again: the REP1 drop-in (cluster march, more than 48 KB at 180
columns) and the two-column tile pass of an odd grid.  Results equal the first
device's bit for bit.  Needs two GPUs.
"""
import ctypes as C

import numpy as np
import pytest

from musoc_solver_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_two():
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two CUDA devices")
    from musoc_solver_b200 import build

    build.build()
    return torch


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def test_rep1_on_both_devices(torch_two):
    from musoc_solver_b200 import native

    torch, L = torch_two, native.lib()
    i2, nb = 180, 15
    ie = np.cumsum(np.full(nb, 6, np.int32)).astype(np.int32) + 1
    j2 = int(ie[-1]) - 1
    p = P.idealised(i2, j2)
    c = [np.ascontiguousarray(a, np.float32) for a in p.coeffs()]
    rng = np.random.default_rng(1)
    rinv, rinv1 = (0.01 * rng.standard_normal((n, i2, i2)) for n in (nb, nb - 1))
    f = rng.standard_normal((j2, i2)).astype(np.float32)
    x0 = rng.standard_normal((j2 + 2, i2 + 2))
    out = []
    for dev in (0, 1, 0):
        with torch.cuda.device(dev):
            x, h = x0.copy(), np.zeros((j2 + 2, i2 + 2))
            d0, d1, d2 = np.zeros((nb - 1, i2)), np.zeros(i2), np.zeros(i2)
            n = [C.byref(C.c_int(v)) for v in (i2 + 2, i2, nb)]
            L.rep1_(*[_p(v) for v in c], _p(rinv), _p(rinv1), _p(d0), _p(d1), _p(d2), _p(f),
                    _p(h), _p(x), _p(ie), *n)
            assert L.sevp_last_status() == 0, dev
            out.append(x)
    assert np.array_equal(out[0], out[1], equal_nan=True)
    assert np.array_equal(out[0], out[2], equal_nan=True)


def test_tile_pass_on_both_devices(torch_two):
    from musoc_solver_b200 import native as N
    from musoc_solver_b200.solver import SevpSolver

    torch = torch_two
    p = P.global_grid(131, 65, seed=3)
    r = np.random.default_rng(2).standard_normal((p.ny, p.nx))
    out = []
    for dev in (0, 1):
        with torch.cuda.device(dev):
            s = SevpSolver(p, tile_m=16, tile_h=16, device=f"cuda:{dev}")
            z = s.precondition(torch.from_numpy(r).to(f"cuda:{dev}"))
            assert s.tile_kernel_used() == N.PASS_B_PAIRS
            out.append(z.cpu().numpy())
            s.close()
    assert np.array_equal(out[0], out[1])
