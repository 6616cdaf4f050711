"""rfgpu_residual_noalloc's FP64 face fluxes, on either kind of products: equal to
rfgpu_residual bit for bit for every flux function and order, at the smallest
region and on both sides of the face count where the products change."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K
from rocflupicl_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 15999, 16000, 16001])   # 8 n - 4 faces
@pytest.mark.parametrize("order", [1, 2])
def test_noalloc_equals_residual(n, order):
    for discr in sorted(K.SCHEME_NAMES):
        num = K.Numerics(spaceDiscr=discr, spaceOrder=order, venkatGuard=1)
        c = K.shock_tube(n, numerics=num)
        assert c.mesh.nFaces == 8 * n - 4
        rng = np.random.default_rng(n)
        c.cv *= 1.0 + 0.1 * rng.random((c.mesh.nCells, 1))
        c.cv[rng.integers(0, c.mesh.nCells, 3), 1] = 1e-200   # beyond the integer products
        c.dv[:] = K.eos_dv(num, c.cv)
        r = E.Region(c)
        ref = r.residual()
        got = r.residual_noalloc()
        r.close()
        assert np.array_equal(got, ref)
