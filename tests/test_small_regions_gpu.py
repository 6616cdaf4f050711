"""Passes chosen by a region's size: at the edges of their tiles and of the
sizes where the choice changes, the default launches equal another launch
shape's bit for bit (gradients, residual, a whole step)."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [K.PREC_FP64, K.PREC_MIXED, K.PREC_SPLIT])
@pytest.mark.parametrize("n", [8, 16, 17, 33, 12799, 12800, 32001])
def test_default_launches_equal_tuned_shape(n, prec):
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_HLLC, venkatGuard=1, precision=prec)
    c = K.shock_tube(n, numerics=num)
    rng = np.random.default_rng(n)
    c.cv *= 1.0 + 0.01 * rng.random((c.mesh.nCells, 1))
    c.dv[:] = K.eos_dv(num, c.cv)
    out = []
    for shape in ({}, {"gradBlock": 256, "faceBlock": 64, "facesPerThread": 2, "cellBlock": 256}):
        r = E.Region(c)
        r.set_tuning(**shape)
        rhs, g = r.residual(), r.gradients()
        r.set_time(1.0)
        r.steps_graph(2, 0.5, 1.0)
        out.append((rhs, g) + r.download() + (np.array(r.time()),))
        r.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
