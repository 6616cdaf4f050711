"""The sizes where a pass changes its kernel, with the last region of one side and
the first of the other: 399 and 400 tiles of 128 cells (the mixed gradient pass
of small regions), 3,996 and 4,000 slices of 32 cells (the FP64 gradient
pass's blocks; 999 and 1,000 tiles).  The default launches equal another launch
shape's bit for bit (gradients, residual, two steps)."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n,tiles", [
    (K.PREC_MIXED, 12768, 399), (K.PREC_MIXED, 12769, 400),
    (K.PREC_SPLIT, 12768, 399), (K.PREC_SPLIT, 12769, 400),
    (K.PREC_FP64, 31968, 999), (K.PREC_FP64, 31969, 1000)])
def test_default_launches_equal_tuned_shape(prec, n, tiles):
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_HLLC, venkatGuard=1, precision=prec)
    c = K.shock_tube(n, numerics=num)
    assert (c.mesh.nCells + 127) // 128 == tiles
    c.cv *= 1.0 + 0.01 * np.random.default_rng(n).random((c.mesh.nCells, 1))
    c.dv[:] = K.eos_dv(num, c.cv)
    out = []
    for shape in ({}, {"gridCap": 200, "gradBlock": 256, "cellBlock": 256}):
        r = E.Region(c)
        r.set_tuning(**shape)
        rhs, g = r.residual(), r.gradients()
        r.set_time(1.0)
        r.steps_graph(2, 0.5, 1.0)
        out.append((rhs, g) + r.download() + (np.array(r.time()),))
        r.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
