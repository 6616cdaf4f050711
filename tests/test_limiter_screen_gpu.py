"""The FP64 limiter's screen against the oracle, bit for bit, where its quotients
leave FP32's normal range: cells at an extremum (the bound is 0) with face
increments of 1e9 and volumes of 1e-22, whose terms volume / (2 d2^2) are
around 1e-40, and nearly symmetric fields, so that two faces' terms often
agree to 1e-7 and only one of them decides."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K
from rocflupicl_gb300 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,amp,noise,seed", [
    (64, 5e-8, 1.6e10, 1e-7, 4),    # one cell's deciding face is lost without the range test
    (32, 1e-8, 1.6e9, 5e-8, 1),
    (32, 1e-8, 1e9, 1e-7, 6),
])
@pytest.mark.parametrize("guard", [0, 1])
def test_tiny_limiters_bitwise(n, h, amp, noise, seed, guard):
    from oracle.oracle import Oracle
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_ROE, venkatGuard=guard)
    m = M.box(M.HEX, n, n, n, hi=(n * h,) * 3)
    i = np.rint(m.cofg / h - 0.5).astype(int)
    rng = np.random.default_rng(seed)
    r, u, v, w, p = (amp * (1 + rng.random((2 * n, n))[i[:, 0] + i[:, 1], i[:, 2]]) *
                     (1 + noise * rng.random(m.nCells)) for _ in range(5))
    cv = K.prim_to_cv(num, r, u, v, w, p)
    with np.errstate(invalid="ignore"):
        dv = K.eos_dv(num, cv)
    dv[:, 0] = p
    c = K.Case("extrema", m, num, [K.PatchBC(K.BC_SLIPWALL, 2) for _ in range(6)], cv, dv)
    g_o = Oracle(c).residual(c.cv, c.dv)[1]
    reg = E.Region(c)
    reg.residual()
    g = reg.gradients()
    reg.close()
    assert np.array_equal(g, g_o)
