"""The mixed path's limiter quotient a * (1/b) and WENO weight 1/b against FP64
division.  The PTX manual bounds the relative error of the approximate
reciprocal by 2^-23; the quotient's product rounds once more, so 2^-23 + 2^-24
and their product."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from rocflupicl_gb300 import _build

pytestmark = pytest.mark.gpu

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "kernels", "reciprocal_check.cu")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("rec") / "reciprocal_check.so")
    subprocess.run([_build._nvcc(), _build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "--expt-relaxed-constexpr", f"-I{_build.INCLUDE}", f"-I{_build.CSRC}",
                    SRC, "-o", lib], check=True)
    f = C.CDLL(lib).reciprocal_check
    fp = C.POINTER(C.c_float)
    f.argtypes, f.restype = [fp, fp, C.c_int, fp, fp], C.c_int

    def run(a, b):
        a, b = (np.ascontiguousarray(x, np.float32) for x in (a, b))
        q, r = np.empty_like(a), np.empty_like(a)
        p = [x.ctypes.data_as(fp) for x in (a, b, q, r)]
        assert f(p[0], p[1], a.size, p[2], p[3]) == 0
        return a.astype(np.float64), b.astype(np.float64), q, r
    return run


def test_error_bounds(check):
    rng = np.random.default_rng(1)
    n = 1 << 20
    e = rng.uniform(-100.0, 120.0, n)       # denominators from 1e-30 to 1e36
    sign = rng.choice([-1.0, 1.0], n)
    b = sign * np.exp2(e) * rng.uniform(1.0, 2.0, n)
    t = np.exp2(rng.uniform(-40.0, 4.0, n))  # the quotients: limiters up to a few
    a, b, q, r = check(t * b, b)
    keep = (np.abs(a) > 1e-37) & (np.abs(a) < 3e38)
    assert keep.mean() > 0.8
    exact = a[keep] / b[keep]
    err = np.abs(q[keep] / exact - 1.0)
    assert err.max() <= 2.0 ** -23 + 2.0 ** -24 + 2.0 ** -47
    assert np.abs(r * b - 1.0).max() <= 2.0 ** -23


def test_edges(check):
    inf, nan = np.inf, np.nan
    a = [1.0, -1.0, 1.0, 0.0, nan, 1.0, 1.0, 0.0]
    b = [1e-12, 1e-12, -1e-12, 1e-12, 1.0, nan, 3e38, 3e38]
    _, _, q, _ = check(a, b)
    assert np.allclose(q[:3], [1e12, -1e12, -1e12], rtol=2e-7)
    assert q[3] == 0.0 and np.isnan(q[4]) and np.isnan(q[5])
    assert q[6] == 0.0 and q[7] == 0.0      # beyond 2^126 the reciprocal flushes to zero
    _, _, q, _ = check([inf, -inf], [1.0, 2.0])
    assert q[0] == inf and q[1] == -inf
