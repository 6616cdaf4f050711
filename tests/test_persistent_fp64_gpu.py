"""FP64 persistent stages (a warp per 32 cells and variable) against one launch
per pass, bit for bit, at the edges of slices, tiles and grids: fewer warps
than slices and variables, as many, and more, with a single block too (one
cell of length has singular moments and NaN gradients)."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reconst", [K.RECONST_LIM_VENKAT, K.RECONST_NONE, K.RECONST_WENO_XYZ])
@pytest.mark.parametrize("n", [1, 8, 9, 33, 972, 973, 4003])
def test_region(n, reconst):
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_HLLC, venkatGuard=1, reconst=reconst)
    c = K.shock_tube(n, numerics=num)
    rng = np.random.default_rng(n)
    c.cv *= 1.0 + 0.01 * rng.random((c.mesh.nCells, 1))
    c.dv[:] = K.eos_dv(num, c.cv)
    out = []
    for shape in ({}, {"persistentStage": 1}, {"persistentStage": 1, "gridCap": 1},
                  {"persistentStage": 1, "gridCap": 7}):
        r = E.Region(c)
        r.set_tuning(**shape)
        r.set_time(1.0)
        for _ in range(2):
            r.step(0.5, 1.0)
        out.append((r.gradients(),) + r.download() + (np.array(r.time()),))
        r.close()
    for got in out[1:]:
        assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(got, out[0]))


def test_batch_of_uneven_regions():
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_ROE, venkatGuard=1)
    cases = K.tube_ensemble(count=7, seed=9, n_min=5, n_max=500, numerics=num)
    out = []
    for coop in (0, 1):
        regs = [E.Region(c) for c in cases]
        for r in regs:
            r.set_time(1.0)
        b = E.Batch(regs)
        b.set_tuning(persistentStage=coop)
        b.steps_graph(3, 0.5, 1e-3)
        b.sync()
        out.append([r.download() + (np.array(r.time()),) for r in regs])
        b.close()
        for r in regs:
            r.close()
    for x, y in zip(*out):
        assert all(np.array_equal(a, b) for a, b in zip(x, y))
