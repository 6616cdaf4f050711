"""Batches on both sides of the size where the FP32-flux passes stop sharing a
launch: the same steps bit for bit as with another face shape, which always
launches the flux passes one by one, and the launches counted."""
import numpy as np
import pytest

from rocflupicl_gb300 import case as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [K.PREC_MIXED, K.PREC_SPLIT, K.PREC_FP64])
@pytest.mark.parametrize("tiles", [49999, 50000])
def test_batch_flux_launches(tiles, prec):
    from rocflupicl_gb300 import engine as E
    num = K.Numerics(spaceDiscr=K.DISCR_UPW_HLLC, venkatGuard=1, precision=prec)
    big = K.shock_tube((tiles - 1) * 16, numerics=num)     # 8 n - 4 faces, 128 a tile
    small = K.shock_tube(9, numerics=num)                  # one tile
    assert sum((c.mesh.nFaces + 127) // 128 for c in (big, small)) == tiles
    out = []
    for shape in ({}, {"faceBlock": 64}):
        regs = [E.Region(c) for c in (big, small)]
        for r in regs:
            r.set_time(1.0)
        b = E.Batch(regs)
        b.set_tuning(**shape)
        n0 = b.launches
        b.step(0.5, 1.0)
        b.sync()
        out.append((b.launches - n0, [r.download() for r in regs], [r.time() for r in regs]))
        b.close()
        for r in regs:
            r.close()
    merged = prec == K.PREC_FP64 or tiles < 50000
    assert out[0][0] == (9 if merged else 13) and out[1][0] == 13
    assert out[0][2] == out[1][2]
    for x, y in zip(out[0][1], out[1][1]):
        assert all(np.array_equal(a, c) for a, c in zip(x, y))
