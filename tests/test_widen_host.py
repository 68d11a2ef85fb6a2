"""widen (widen.cuh), the conversion of a float to a double by integer
instructions, compiled as host C++: the double of every float tried, zeros of both
signs, subnormals, infinities and NaN among them."""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from test_fp64_helpers_host import CSRC, CUDA_INC, SHIM

EXTRA = r"""
inline unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
inline double __hiloint2double(int hi, int lo)
{
    return __longlong_as_double((long long)(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo));
}
using std::fabs;
"""
DRIVER = r"""
#include "widen.cuh"
extern "C" void h_widen(const float* x, long n, double* out) { for (long i = 0; i < n; ++i) out[i] = lat::widen(x[i]); }
"""


def test_widen_is_the_conversion(tmp_path):
    gxx = shutil.which("g++")
    if not gxx or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "shim.h").write_text(SHIM + EXTRA)
    (tmp_path / "drv.cpp").write_text('#include "shim.h"\n' + DRIVER)
    so = tmp_path / "libwiden.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CUDA_INC}", f"-I{CSRC}",
                    str(tmp_path / "drv.cpp"), "-o", str(so)], check=True, capture_output=True)
    rng = np.random.default_rng(2)
    bits = rng.integers(0, 1 << 32, 500_000, dtype=np.uint64).astype(np.uint32)
    edges = np.array([0, 1, 2, 0x7fffff, 0x800000, 0x800001, 0x3f800000, 0x7f7fffff, 0x7f800000, 0x7fc00000, 0x7f800001], np.uint32)
    bits = np.concatenate([bits, bits & np.uint32(0x807fffff), edges, edges | np.uint32(1 << 31)])
    x = bits.view(np.float32)
    out = np.empty(x.size)
    P = ctypes.c_void_p
    ctypes.CDLL(str(so)).h_widen(P(x.ctypes.data), ctypes.c_long(x.size), P(out.ctypes.data))
    nan = np.isnan(x)
    assert np.isnan(out[nan]).all()
    assert np.array_equal(out[~nan].view(np.uint64), x[~nan].astype(np.float64).view(np.uint64))
