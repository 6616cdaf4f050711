"""Transfers of regions whose cell counts lie at the edges of the chunk counts
(one chunk, two, six and eight): the host-resident step equals upload, step
and download bit for bit, and an upload comes back as it went up."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [K.PREC_MIXED, K.PREC_SPLIT])
@pytest.mark.parametrize("dims", [(28, 28, 28), (43, 35, 29), (64, 64, 33), (76, 68, 68)])
def test_step_host_equals_three_calls_over_chunk_counts(dims, prec):
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_HLLC, venkatGuard=1, precision=prec)
    c = K.tet_shock_box(dims[0], ny=dims[1], nz=dims[2], numerics=num)
    a = E.Region(c)
    cv, dv = a.download()
    assert np.allclose(cv, c.cv, rtol=1e-13, atol=0.0)  # the float-float pair's 48 bits
    a.upload(c.cv)  # p from the conserved state, as the host-resident step forms it
    a.set_time(1.0)
    a.step(0.5, 1.0)
    cv, dv = a.download()
    a.close()
    b = E.Region(c)
    b.set_time(1.0)
    cvh, dvh = np.ascontiguousarray(c.cv).copy(), np.empty_like(c.dv)
    b.step_host(cvh, dvh, 0.5, 1.0)
    b.close()
    assert np.array_equal(cvh, cv)
    assert np.array_equal(dvh, dv)
