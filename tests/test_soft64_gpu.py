"""Products of the FP64 gradient pass formed on the integer pipes, and its
screened limiter: bit equality with the oracle where they can go wrong - short
significands (rounding ties, exact products, equal limiter terms), zeros of
both signs, magnitudes outside the integer products' exponent range,
infinities and NaNs - on meshes with and without zero weights."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu


def states(kind, c, rng):
    N = c.mesh.nCells
    r = 1.0 + 0.2 * rng.random(N)
    u, v, w = (100.0 * (rng.random(N) - 0.5) for _ in range(3))
    p = 1.0e5 * (1.0 + 0.2 * rng.random(N))
    if kind == "short":      # few significant bits: ties and exact products
        r, p = np.round(r * 16) / 16, np.round(p / 4096) * 4096
        u, v, w = np.round(u), np.round(v / 8) * 8, np.zeros(N)
    elif kind == "layered":  # a one-dimensional field: equal differences across faces
        x = c.mesh.cofg[:, 0]
        r, u, v, w, p = 1.0 + x, 10.0 * x, np.zeros(N), -np.zeros(N), 1.0e5 * (1.0 + 0.1 * x)
    elif kind == "tiny":     # differences around and below the exponent range
        u, v, w = u * 1e-155, v * 1e-160, w * 1e-290
    elif kind == "wide":
        u, v = u * 10.0 ** rng.integers(-30, 4, N), v * 10.0 ** rng.integers(-170, 2, N)
    elif kind == "special":
        p[rng.integers(0, N, 3)] = np.inf
        u[rng.integers(0, N, 3)] = np.nan
        v[rng.integers(0, N, 3)] = -np.nan
    return K.prim_to_cv(c.numerics, r, u, v, w, p)


@pytest.mark.parametrize("kind", ["random", "short", "layered", "tiny", "wide", "special"])
@pytest.mark.parametrize("mesh", ["tube", "tet", "box"])
def test_fp64_gradients_and_residual_bitwise(mesh, kind):
    from oracle.oracle import Oracle
    from rocflupicl_gb300 import engine as E
    for guard in (0, 1):
        num = K.Numerics(spaceDiscr=K.DISCR_UPW_ROE, venkatGuard=guard)
        c = (K.shock_tube(37, numerics=num) if mesh == "tube" else
             K.tet_shock_box(5, numerics=num) if mesh == "tet" else K.mixed_box(6, numerics=num))
        with np.errstate(all="ignore"):
            c.cv[:] = states(kind, c, np.random.default_rng(5))
            c.dv[:] = K.eos_dv(num, c.cv)
            rhs_o, g_o = Oracle(c).residual(c.cv, c.dv)
        reg = E.Region(c)
        rhs, g = reg.residual(), reg.gradients()
        reg.close()
        assert np.array_equal(g, g_o, equal_nan=True)
        assert np.array_equal(rhs, rhs_o, equal_nan=True)
