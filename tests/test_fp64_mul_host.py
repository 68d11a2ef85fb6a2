"""The integer product of fp64_exact.cuh (factor, mul), compiled from its CUDA
header as host C++: bitwise the IEEE product a*b for every operand in its
range, exact ties and near-ties of the rounding, carries, products on both
sides of a power of two; zeros, subnormals, large values, Inf and NaN are told
apart by product_range."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "axions_gb300" / "csrc"
CUDA_INC = Path("/usr/local/cuda/include")

SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>
#undef __device__
#undef __forceinline__
#undef __noinline__
#define __device__
#define __forceinline__ inline
#define __noinline__ inline
inline double __dmul_rn(double a, double b) { return a * b; }
inline long long __double_as_longlong(double x) { long long u; std::memcpy(&u, &x, 8); return u; }
inline double __longlong_as_double(long long u) { double x; std::memcpy(&x, &u, 8); return x; }
"""

DRIVER = r"""
#include "fp64_exact.cuh"
extern "C" void h_mul(const double* a, const double* b, long n, double* out, double* ref, int* range) {
    for (long i = 0; i < n; ++i) {
        const unsigned x = lat::product_range(a[i]), y = lat::product_range(b[i]);
        const bool in = (x > y ? x : y) < lat::kProductSpan;
        ref[i] = a[i] * b[i];
        out[i] = in ? lat::mul(lat::factor(a[i]), lat::factor(b[i])) : ref[i];
        range[i] = in;
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("mul")
    (d / "shim.h").write_text(SHIM)
    (d / "drv.cpp").write_text(DRIVER)
    so = d / "libmul.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CUDA_INC}", f"-I{CSRC}",
                    "-include", str(d / "shim.h"), str(d / "drv.cpp"), "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def check(lib, a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    got, ref, inr = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.int32)
    P = ctypes.c_void_p
    lib.h_mul(P(a.ctypes.data), P(b.ctypes.data), ctypes.c_long(a.size), P(got.ctypes.data), P(ref.ctypes.data),
              P(inr.ctypes.data))
    x, y = np.abs(a), np.abs(b)
    want = (x >= 2.0 ** -510) & (x < 2.0 ** 512) & (y >= 2.0 ** -510) & (y < 2.0 ** 512)
    assert np.array_equal(inr != 0, want)
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(got), nan)
    bad = (got.view(np.uint64) != ref.view(np.uint64)) & ~nan
    assert not bad.any(), (a[bad][:3], b[bad][:3], got[bad][:3], ref[bad][:3])


def doubles(rng, n, emin, emax, mant=None):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64) if mant is None else mant
    return ((rng.integers(1023 + emin, 1024 + emax, n, dtype=np.uint64) << np.uint64(52)) | m |
            (rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63))).view(np.float64)


def test_product_is_the_ieee_product(lib):
    rng = np.random.default_rng(17)
    n = 2_000_000
    check(lib, doubles(rng, n, -3, 3), doubles(rng, n, -3, 3))
    check(lib, doubles(rng, n, -600, 600), doubles(rng, n, -600, 600))
    check(lib, doubles(rng, n, -1022, 1023), doubles(rng, n, -1022, 1023))
    # few significant bits: exact products and exact ties; all-ones mantissas: carries
    for bits in (1, 5, 20, 26, 27, 28, 40):
        mask = np.uint64(((1 << bits) - 1) << (52 - bits))
        ma = rng.integers(0, 1 << 52, n // 4, dtype=np.uint64) & mask
        mb = rng.integers(0, 1 << 52, n // 4, dtype=np.uint64) & np.uint64(((1 << min(52, 54 - bits)) - 1) << (52 - min(52, 54 - bits)))
        check(lib, doubles(rng, n // 4, -2, 2, ma), doubles(rng, n // 4, -2, 2, mb))
        ones = np.uint64((1 << 52) - 1) - (rng.integers(0, 1 << bits, n // 4, dtype=np.uint64))
        check(lib, doubles(rng, n // 4, -2, 2, ones), doubles(rng, n // 4, -2, 2))
        check(lib, doubles(rng, n // 4, -2, 2, ones), doubles(rng, n // 4, -2, 2, ones[::-1].copy()))
    special = np.array([0.0, -0.0, 5e-324, -5e-324, 2.2250738585072014e-308, 1.7976931348623157e308, np.inf, -np.inf, np.nan,
                        1.0, -1.0, 2.0 ** -510, 2.0 ** 512, np.nextafter(2.0 ** 512, 0), np.nextafter(2.0 ** -510, 0), 0.5, 3.0])
    x, y = np.meshgrid(special, special)
    check(lib, x.ravel(), y.ravel())
