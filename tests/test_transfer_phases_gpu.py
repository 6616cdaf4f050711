"""The host-resident step over two and more transfer chunks, whose first stage
runs its gradient pass and whose last stage runs every pass in phases: equal to
upload + step + download bit for bit, for the schemes, integrators, precisions
and numberings that take different phases (one stage or several, WENO without
phased gradients, no limiter).  The chunk count of each size is read off the
conversions that an upload launches, one per chunk."""
import functools

import numpy as np
import pytest

from rocflupicl_gb300 import case as K
from rocflupicl_gb300 import engine as E

pytestmark = pytest.mark.gpu

VARIANTS = {
    "roe-wray": dict(spaceDiscr=K.DISCR_UPW_ROE),
    "hllc-rk4": dict(spaceDiscr=K.DISCR_UPW_HLLC, rkScheme=K.RK_SCHEME_4_CLASSICAL),
    "ausm+-euler": dict(spaceDiscr=K.DISCR_UPW_AUSMPLUS, rkScheme=K.RK_SCHEME_1_EULER),
    "ausm+up-unlimited": dict(spaceDiscr=K.DISCR_UPW_AUSMPLUSUP, reconst=K.RECONST_NONE),
    "weno": dict(spaceDiscr=K.DISCR_UPW_ROE, reconst=K.RECONST_WENO_XYZ),
    "split": dict(spaceDiscr=K.DISCR_UPW_ROE, precision=K.PREC_SPLIT),
    "split-rk4": dict(spaceDiscr=K.DISCR_UPW_HLLC, rkScheme=K.RK_SCHEME_4_CLASSICAL,
                      precision=K.PREC_SPLIT),
}


@functools.lru_cache(maxsize=1)
def box(dims):
    return K.tet_shock_box(dims[0], ny=dims[1], nz=dims[2], seed=7, Ms=1.2)  # weak: unlimited too


@pytest.mark.parametrize("chunks,dims", [
    (1, (44, 35, 28)), (2, (44, 35, 29)), (3, (41, 41, 40)), (4, (45, 45, 44)),
    (5, (48, 48, 48)), (6, (51, 51, 51)), (8, (71, 71, 70)),
    (7, (54, 54, 54)), (8, (59, 59, 59))])   # here the step itself runs in 6
@pytest.mark.parametrize("order", [E.ORDER_HOST, E.ORDER_LOCALITY])
@pytest.mark.parametrize("variant", sorted(VARIANTS))
def test_phased_step_equals_three_calls(chunks, dims, order, variant):
    c = box(dims)
    num = K.Numerics(**{**dict(precision=K.PREC_MIXED, venkatGuard=1), **VARIANTS[variant]})
    r = E.Region(K.Case(c.name, c.mesh, num, c.bcs, c.cv, c.dv), cell_order=order)
    n0 = r.launches
    r.upload(c.cv)
    assert r.launches - n0 == chunks
    r.set_time(0.0)
    dt = r.time_step(0.4, 1.0, 0.0, 1.0)
    r.set_time(0.0)
    cv = np.ascontiguousarray(c.cv).copy()
    for _ in range(2):
        r.upload(cv)
        r.step(0.4, dt)
        cv, dv = r.download()
    t = r.time()
    r.set_time(0.0)
    cvh, dvh = E.PinnedArray(cv.shape), E.PinnedArray(dv.shape)
    cvh.array[:] = c.cv
    for _ in range(2):
        r.step_host(cvh.array, dvh.array, 0.4, dt)
    assert np.all(np.isfinite(cv)) and not np.array_equal(cv, c.cv)
    assert np.array_equal(cvh.array, cv)
    assert np.array_equal(dvh.array, dv)
    assert r.time() == t and r.status() == 0
    cvh.close()
    dvh.close()
    r.close()
