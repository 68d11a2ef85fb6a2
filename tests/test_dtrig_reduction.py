"""The fixed-point sine and cosine of dtrig.cuh, compiled as host C++: its constants
against exact fractions, and its results where the reduction changes: at quadrant
boundaries, at both sides of the 2^-20 about a multiple of pi/2 inside which CUDA's
functions are called, of 2^16 from which they are, and of 2^-27 below which sin x = x.
Within the 1.65 ulps that the header derives."""
import ctypes
import re
import shutil
import subprocess
from fractions import Fraction
from math import factorial

import numpy as np
import pytest

from test_fp64_helpers_host import CSRC, CUDA_INC, SHIM

PI = Fraction(314159265358979323846264338327950288419716939937510582097494459230781640628620899862803482534211706798214808651,
              10 ** 110)

DRIVER = r"""
#include "dtrig.cuh"
extern "C" void h_trig(const double* x, long n, double* out)
{
    for (long i = 0; i < n; ++i) {
        double s, c;
        lat::dsincos(x[i], &s, &c);
        out[i] = lat::dsin(x[i]); out[n + i] = s; out[2 * n + i] = c;
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("reduction")
    (d / "shim.h").write_text(SHIM)
    (d / "drv.cpp").write_text('#include "shim.h"\n' + DRIVER)
    so = d / "libreduction.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CUDA_INC}", f"-I{CSRC}",
                    str(d / "drv.cpp"), "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def test_constants():
    text = (CSRC / "dtrig.cuh").read_text()
    assert abs(PI - Fraction(355, 113)) < Fraction(1, 10 ** 6)
    p1, p2 = (Fraction(float.fromhex(re.search(rf"kP{k} = (0x[0-9a-fp.+-]+)", text).group(1))) for k in (1, 2))
    assert p1.numerator.bit_length() <= 36 and abs(p1 + p2 - PI / 2) < Fraction(1, 2 ** 92)
    for name, first in (("S", 1), ("C", 0)):
        for n in range(1, 10):
            value = int(re.search(rf"k{name}{n} = (0x[0-9a-f]+)", text).group(1), 16)
            unit = 2 ** (64 if n <= 5 else 60)
            assert abs(value - Fraction(unit, factorial(2 * n + first))) <= Fraction(1, 2), (name, n)


def test_where_the_reduction_changes(lib):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("needs a long double of 64 bits")
    rng = np.random.default_rng(6)
    half_pi = np.longdouble(np.pi / 2) + np.longdouble(6.123233995736766e-17)
    k = np.concatenate([np.arange(-300, 301), rng.integers(-41721, 41722, 4000)])
    off = np.concatenate([[0.0], 2.0 ** -np.arange(1.0, 60.0), 2.0 ** -20 * (1 + np.linspace(-1e-3, 1e-3, 21)), [np.pi / 4]])
    off = np.concatenate([off, -off])
    x = [(k[:, None] * half_pi + off).astype(np.float64).ravel()]
    edges = np.array([2.0 ** 16, 2.0 ** -27, 2.0 ** -20, np.pi / 4, np.pi / 2, 1.0])
    x.append((edges[:, None] + np.spacing(edges)[:, None] * np.arange(-40, 41)).ravel())
    x.append(rng.uniform(-65536, 65536, 200_000))
    x.append(10.0 ** rng.uniform(-12, 0, 100_000))
    x = np.concatenate(x)
    x = np.ascontiguousarray(np.concatenate([x, -x]))
    out = np.zeros((3, x.size))
    P = ctypes.c_void_p
    lib.h_trig(P(x.ctypes.data), ctypes.c_long(x.size), P(out.ctypes.data))
    xl = x.astype(np.longdouble)
    for got, want in ((out[0], np.sin(xl)), (out[1], np.sin(xl)), (out[2], np.cos(xl))):
        ulp = np.spacing(np.abs(want.astype(np.float64)))
        assert (np.abs(got - want) <= 1.65 * ulp).all(), float(np.max(np.abs(got - want) / ulp))
    assert np.array_equal(out[0], out[1])
