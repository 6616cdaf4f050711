"""FP64 residuals, gradients, stages and status bits against the oracle, bit for
bit, on states whose operands leave the range of the integer products: every
flux function at both orders, the RK update under Wray and classical RK4, the
EOS, and the gate of AfterUpdateMP's checks on both sides (pressures that are
cancellation residues of the energy, positive and negative)."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu

KINDS = ["random", "zeros", "tiny", "wide", "huge", "special", "residue", "negative"]


def states(kind, num, mesh, rng):
    N = mesh.nCells
    r = 1.0 + 0.2 * rng.random(N)
    u, v, w = (100.0 * (rng.random(N) - 0.5) for _ in range(3))
    p = 1.0e5 * (1.0 + 0.2 * rng.random(N))
    if kind == "zeros":
        u, v, w = np.where(rng.random(N) < 0.5, 0.0, -0.0), np.where(rng.random(N) < 0.5, v, -0.0), 0 * w
    elif kind == "tiny":
        u, v, w = u * 1e-155, v * 1e-160, w * 1e-290
    elif kind == "wide":
        u, v = u * 10.0 ** rng.integers(-30, 4, N), v * 10.0 ** rng.integers(-170, 2, N)
    elif kind == "huge":
        i = rng.integers(0, N, 5)
        r[i], u[i[:3]], p[i[2:]] = 1e160, 1e80, 1e200
    cv = K.prim_to_cv(num, r, u, v, w, p)
    if kind == "special":
        cv[rng.integers(0, N, 2), 4] = np.inf
        cv[rng.integers(0, N, 2), 1] = np.nan
        cv[rng.integers(0, N, 2), 2] = -np.inf
        cv[rng.integers(0, N, 2), 0] = 5e-324
    elif kind in ("residue", "negative"):
        kin = 0.5 * (cv[:, 1] ** 2 + cv[:, 2] ** 2 + cv[:, 3] ** 2) / cv[:, 0]
        i = rng.random(N) < 0.3
        e = 10.0 ** rng.uniform(-17.0, -6.0, N)
        if kind == "negative":
            e = e * rng.choice([-1.0, 1.0], N)
        cv[i, 4] = (kin * (1.0 + e))[i]
    return cv


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    bits = a.view(np.int64) == b.view(np.int64)
    return bool(np.all(bits | (np.isnan(a) & np.isnan(b)) | ((a == 0.0) & (b == 0.0))))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("scheme", sorted(K.SCHEME_NAMES))
@pytest.mark.parametrize("mesh", ["tube", "tet"])
def test_stages_bitwise(mesh, scheme, kind):
    from oracle.oracle import Oracle
    from rocflupicl_gb300 import engine as E
    for order in (2, 1):
        for rk in (K.RK_SCHEME_3_WRAY, K.RK_SCHEME_4_CLASSICAL):
            num = K.Numerics(spaceDiscr=scheme, spaceOrder=order, rkScheme=rk)
            c = K.shock_tube(37, numerics=num) if mesh == "tube" else K.tet_shock_box(5, numerics=num)
            with np.errstate(all="ignore"):
                c.cv[:] = states(kind, num, c.mesh, np.random.default_rng(order + 10 * rk))
                c.dv[:] = K.eos_dv(num, c.cv)
                cv, dv = c.cv.copy(), c.dv.copy()
                orc = Oracle(c)
                reg = E.Region(c)
                rhs_o, g_o = orc.residual(cv, dv)
                assert same(reg.residual(), rhs_o) and same(reg.gradients(), g_o)
                for stage in range(1, reg.nSteps + 1):
                    st_o = orc.stage(cv, dv, stage, 1e-7)
                    reg.rk_stage(stage, 1e-7)
                    cvg, dvg = reg.download()
                    assert same(cvg, cv) and same(dvg, dv), (order, rk, stage)
                    assert reg.status() == st_o, (order, rk, stage)
                reg.close()
