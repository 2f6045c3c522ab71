"""REP1 and REP at the sizes where the cluster's marching solve can go wrong:
fewer columns than CTAs, column counts that do not divide by the CTAs or the
mat-vec's batch, one- and two-row blocks, a last block of another height, and
a grid whose rows do not fit the cluster's shared memory (the one-CTA kernel
runs).  X and every workspace (H, DUM0, DUM1, DUM2) equal the CPU oracle's
restatement of the reference bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

from musoc_solver_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from musoc_solver_b200 import build, native

    build.build()
    return native.lib()


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _i(v):
    return C.byref(C.c_int(int(v)))


# (columns, block heights; the first block has one equation row less)
CASES = [
    (5, [3, 2, 3]),
    (16, [2, 1, 1, 2]),
    (33, [6, 5, 6, 4]),
    (100, [7]),
    (181, [6] * 9 + [5]),
    (260, [6] * 30),  # the rows exceed the cluster's shared memory
]


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("i2,heights", CASES)
def test_march_matches_oracle(L, oracle, i2, heights, periodic):
    ie = np.cumsum(np.array(heights, np.int32)).astype(np.int32) + 1
    j2, nb = int(ie[-1]) - 1, len(heights)
    p = P.idealised(i2, j2)
    p.ac[:] += np.float32(0.05)
    if not periodic:
        p.al[:, 0] = 0.0
        p.ar[:, -1] = 0.0
    c = [np.ascontiguousarray(a, np.float32) for a in p.coeffs()]
    rng = np.random.default_rng(i2)
    # any matrices do: the marching is compared, not its accuracy
    rinv = 0.01 * rng.standard_normal((nb, i2, i2))
    rinv1 = 0.01 * rng.standard_normal((max(nb - 1, 1), i2, i2))
    f = rng.standard_normal((j2, i2)).astype(np.float32)
    x0 = rng.standard_normal((j2 + 2, i2 + 2))
    out = []
    for fn in (L.rep1_ if periodic else L.rep_, None):
        a = dict(d0=np.zeros((max(nb - 1, 1), i2)), d1=np.zeros(i2), d2=np.zeros(i2),
                 h=np.full((j2 + 2, i2 + 2), 7.0), x=x0.copy())
        if fn is not None:
            fn(*[_p(v) for v in c], _p(rinv), _p(rinv1), _p(a["d0"]), _p(a["d1"]), _p(a["d2"]),
               _p(f), _p(a["h"]), _p(a["x"]), _p(ie), _i(i2 + 2), _i(i2), _i(nb))
            assert L.sevp_last_status() == 0
        else:
            ref = oracle.lib().or_rep1 if periodic else oracle.lib().or_rep
            ref(*c, rinv, rinv1, a["d0"], a["d1"], a["d2"], f, a["h"], a["x"], ie, i2 + 2, i2, nb)
        out.append(a)
    for k in ("x", "h", "d0", "d1", "d2"):
        g, o = out[0][k], out[1][k]
        if k == "d0" and nb == 1:
            continue  # not used
        assert np.array_equal(g, o, equal_nan=True), (k, np.abs(g - o).max())
