"""AfterUpdateMP's pressure clamp on cells whose pressure is a cancellation
residue: the EOS forms p = (g-1) rho (E/rho - (1/rho)^2 |m|^2 / 2), the checks
form |u|^2 from the velocities, and the two can differ in sign.  The states
here have a positive EOS pressure and a non-positive one in the checks, with
E/rho - |u|^2/2 as two operations or as one FMA, so every cell has to be
clamped: E becomes rho (1e-12 / (rho (g-1)) + |u|^2 / 2) (libflu/
RFLU_EnforceBounds.F90:163-232)."""
from fractions import Fraction

import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu


def residues(count, rng):
    def fma(a, b, c):
        return float(Fraction(a) * Fraction(b) + Fraction(c))

    out = []
    while len(out) < count:
        n = 20000
        r, m = rng.uniform(0.3, 3.0, n), rng.uniform(0.3, 3.0, n)
        e = 0.5 * m * m / r
        e = e + np.spacing(e) * rng.integers(-3, 4, n)
        ir = 1.0 / r
        u = ir * m
        k_eos, k_chk = 0.5 * ((ir * ir) * (m * m)), 0.5 * (u * u)
        for i in np.where((ir * e - k_eos > 0.0) & (ir * e - k_chk <= 0.0))[0]:
            if fma(ir[i], e[i], -k_eos[i]) > 0.0 and fma(ir[i], e[i], -k_chk[i]) <= 0.0:
                out.append((r[i], m[i], e[i]))
    return np.array(out[:count])


@pytest.mark.parametrize("prec", [K.PREC_FP64, K.PREC_SPLIT])
@pytest.mark.parametrize("rk", [K.RK_SCHEME_3_WRAY, K.RK_SCHEME_4_CLASSICAL, K.RK_SCHEME_1_EULER])
def test_residual_pressure_is_clamped(prec, rk):
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_AUSMPLUS, spaceOrder=1, rkScheme=rk, precision=prec)
    c = K.shock_tube(8, numerics=num)
    n = c.mesh.nCells
    s = residues(n, np.random.default_rng(3))
    c.cv[:] = np.stack([s[:, 0], s[:, 1], np.zeros(n), np.zeros(n), s[:, 2]], axis=1)
    c.dv[:] = K.eos_dv(num, c.cv)
    assert np.all(c.dv[:, 0] > 0.0)
    reg = E.Region(c)
    reg.upload(c.cv)
    reg.rk_stage(1, 0.0)  # no time: the checks alone can change the state
    cv, st = reg.download()[0], reg.status()
    reg.close()
    assert st == E.ST_PCLAMP
    assert np.array_equal(cv[:, :4], c.cv[:, :4])
    u = c.cv[:, 1] / c.cv[:, 0]
    want = c.cv[:, 0] * (1e-12 / (c.cv[:, 0] * (num.gamma_gv - 1.0)) + 0.5 * u * u)
    assert np.all(cv[:, 4] > c.cv[:, 4])
    assert np.all(np.abs(cv[:, 4] - want) <= 8 * np.spacing(want))  # a few roundings of E
