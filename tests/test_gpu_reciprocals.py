"""fast_rcp, fast_rsqrt and fast_sqrt of the explicit path (GPU) against 64-bit division and square
root: every binade of the fast range, its edges, and what lies outside of it.

Bounds: the hardware's seeds are good to 2^-20, the third-order steps leave 2^-59; what is
left are roundings: 1/x one (half an ulp), 1/sqrt(x) the rounding of x y (half of it reaches the
result) and the last one, sqrt(x) the product's besides.  In units of 2^-52 of the value: below
1, 2 and 3.  Outside the fast range the plain operations are taken."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from bes_gb300 import build as nbuild

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
LO, HI = 2.0 ** -1000, 2.0 ** 1000


@pytest.fixture(scope="module")
def reciprocals(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("reciprocals") / "reciprocals.so")
    subprocess.run([nbuild.nvcc(), *nbuild.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-shared",
                    "-Xcompiler", "-fPIC", "-I" + os.path.join(nbuild.ROOT, "include"),
                    os.path.join(HERE, "reciprocals", "reciprocals.cu"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    D = ctypes.POINTER(ctypes.c_double)
    L.reciprocals.argtypes = [D, ctypes.c_int64, D]

    def call(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out = np.zeros((3, x.size))
        assert L.reciprocals(x.ctypes.data_as(D), x.size, out.ctypes.data_as(D)) == 0
        return out

    return call


def test_fast_range(reciprocals):
    rng = np.random.default_rng(0)
    e = np.repeat(np.arange(-1000, 1000), 64)
    x = np.concatenate([np.ldexp(1.0 + rng.random(e.size), e), np.ldexp(rng.uniform(1, 2, 400000), rng.integers(-60, 60, 400000)),
                        [LO, np.nextafter(LO, 1), HI, np.nextafter(HI, 0), 1.0, np.nextafter(1.0, 0), np.nextafter(1.0, 2)]])
    rcp, rsqrt, sqrt = reciprocals(x)
    xl = x.astype(np.longdouble)
    ulp = 2.0 ** -52
    assert (np.abs(rcp * xl - 1) <= ulp).all()
    assert (np.abs(rsqrt * np.sqrt(xl) - 1) <= 2 * ulp).all()
    assert (np.abs(sqrt / np.sqrt(xl) - 1) <= 3 * ulp).all()


def test_outside_the_fast_range(reciprocals):
    x = np.array([0.0, -0.0, 5e-324, 2.0 ** -1060, 2.0 ** -1022, np.nextafter(LO, 0), np.nextafter(HI, np.inf) * 2,
                  2.0 ** 1023, np.finfo(float).max, np.inf, -np.inf, np.nan, -5e-324, -LO, -1.0, -3.7, -HI])
    rcp, rsqrt, sqrt = reciprocals(x)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(rcp, 1.0 / x)
        np.testing.assert_array_equal(rsqrt, 1.0 / np.sqrt(x))
        np.testing.assert_array_equal(sqrt, np.sqrt(x))
