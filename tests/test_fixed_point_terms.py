"""The Laplacian and current of the fused FP64 update in fixed point
(fixed_point.cuh), compiled from its CUDA header as host C++, against long
double: within the bound of its truncations (2^-58 of the largest scalar each),
on the average no further off than the same terms in doubles with one rounding
per operation; zeros and uniform states without a gauge field are exact;
subnormal, huge, infinite and NaN scalars and NaN links are refused."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "axions_gb300" / "csrc"
CUDA_INC = Path("/usr/local/cuda/include")

SRC = r"""
#include "fixed_point.cuh"
#include <cmath>
using namespace lat;
template <class T> static void terms(const T* v, const T* th, T* u, T* cur)
{
    for (int k = 0; k < 2; ++k) u[k] = -6 * v[k];
    for (int a = 0; a < 3; ++a) {
        const T c = th[2 * a], s = th[2 * a + 1], cm = th[6 + 2 * a], sm = th[7 + 2 * a];
        const T* f = v + 2 + 2 * a; const T* b = v + 8 + 2 * a;
        const T A = c * f[0] + s * f[1], B = c * f[1] - s * f[0];
        u[0] += A + (cm * b[0] - sm * b[1]);
        u[1] += B + (cm * b[1] + sm * b[0]);
        cur[a] = v[1] * A - v[0] * B;
    }
}
extern "C" void h_terms(const double* v, const double* link, long n, double* got, double* dbl, double* exact_hi, double* exact_lo,
                        int* ok)
{
    for (long i = 0; i < n; ++i, v += 14, link += 12, got += 5, dbl += 5, exact_hi += 5, exact_lo += 5) {
        double p[2] = {v[0], v[1]}, f[3][2], b[3][2], u[2] = {0, 0}, cur[3] = {0, 0, 0};
        int64_t cs[3], sn[3], csm[3], snm[3];
        for (int a = 0; a < 3; ++a) {
            for (int k = 0; k < 2; ++k) f[a][k] = v[2 + 2 * a + k], b[a][k] = v[8 + 2 * a + k];
            cs[a] = fix::link_of(link[2 * a]), sn[a] = fix::link_of(link[2 * a + 1]);
            csm[a] = fix::link_of(link[6 + 2 * a]), snm[a] = fix::link_of(link[7 + 2 * a]);
        }
        ok[i] = fix::scalar_terms(p, f, b, cs, sn, csm, snm, u, cur);
        for (int k = 0; k < 5; ++k) got[k] = k < 2 ? u[k] : cur[k - 2];
        double du[2], dc[3];
        terms<double>(v, link, du, dc);
        long double lv[14], ll[12], lu[2], lc[3];
        for (int k = 0; k < 14; ++k) lv[k] = v[k];
        for (int k = 0; k < 12; ++k) ll[k] = link[k];
        terms<long double>(lv, ll, lu, lc);
        for (int k = 0; k < 5; ++k) {
            dbl[k] = k < 2 ? du[k] : dc[k - 2];
            const long double e = k < 2 ? lu[k] : lc[k - 2];
            exact_hi[k] = (double)e;
            exact_lo[k] = (double)(e - (long double)exact_hi[k]);
        }
    }
}
extern "C" void h_link(const double* v, long n, double* out) { for (long i = 0; i < n; ++i) out[i] = fix::link_value(fix::link_of(v[i])); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("fixed")
    (d / "drv.cpp").write_text(SRC)
    so = d / "libfixed.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CUDA_INC}", f"-I{CSRC}",
                    str(d / "drv.cpp"), "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def run(lib, v, link):
    v, link = np.ascontiguousarray(v, np.float64), np.ascontiguousarray(link, np.float64)
    n = len(v)
    out = [np.zeros((n, 5)) for _ in range(4)]
    ok = np.zeros(n, np.int32)
    P = ctypes.c_void_p
    lib.h_terms(P(v.ctypes.data), P(link.ctypes.data), ctypes.c_long(n), *[P(o.ctypes.data) for o in out], P(ok.ctypes.data))
    got, dbl, hi, lo = out
    return ok != 0, got, (got - hi) - lo, (dbl - hi) - lo, hi


def links(rng, n, width):
    th = rng.uniform(-width, width, (n, 6))
    return np.stack([np.cos(th), np.sin(th)], -1).reshape(n, 12)


@pytest.mark.parametrize("width", [0.0, 1e-6, 0.3, 4.0])
@pytest.mark.parametrize("scale", [1.0, 1.99, 1e-120, 3e120])
@pytest.mark.parametrize("spread", ["phases", "vacuum", "ranges"])
def test_terms_against_long_double(lib, width, scale, spread):
    rng = np.random.default_rng(4)
    n = 40000
    ph = rng.uniform(0, 2 * np.pi, (n, 7)) if spread != "vacuum" else rng.uniform(0, 2 * np.pi, (n, 1)) + rng.normal(0, 0.1, (n, 7))
    mag = np.exp2(rng.uniform(-40, 0, (n, 7))) if spread == "ranges" else rng.uniform(0.7, 1.3, (n, 7))
    v = (scale * mag[..., None] * np.stack([np.cos(ph), np.sin(ph)], -1)).reshape(n, 14)
    ok, got, err, derr, exact = run(lib, v, links(rng, n, width))
    assert ok.all()
    top = np.abs(v).max(1)[:, None]
    unit = np.concatenate([top, top, top ** 2, top ** 2, top ** 2], 1)
    # 24 products and 14 values truncated, links to 2^-62; the last rounding
    assert (np.abs(err) <= 40 * 2.0 ** -58 * unit + 2.0 ** -53 * np.abs(exact)).all()
    for k in (slice(0, 2), slice(2, 5)):
        assert np.sqrt(np.mean((err[:, k] / unit[:, k]) ** 2)) <= np.sqrt(np.mean((derr[:, k] / unit[:, k]) ** 2)) + 2.0 ** -58


def test_exact_and_refused(lib):
    rng = np.random.default_rng(5)
    one = np.tile([1.0, 0.0], (64, 6))
    v = np.tile(rng.uniform(-1, 1, (64, 2)), (1, 7))
    ok, got, *_ = run(lib, v, one)
    assert ok.all() and (got == 0).all()       # a uniform scalar without a gauge field
    v[:, 3] = 0.0
    ok, got, err, *_ = run(lib, v, one)
    assert ok.all() and (err[:, :2] == 0).all()
    for bad in (0.0, 5e-324, 2.0 ** -500, 2.0 ** 500, np.inf, np.nan):
        w = rng.uniform(-1, 1, (64, 14)) if abs(bad) > 1 or bad != bad else np.zeros((64, 14))
        w[np.arange(64), rng.integers(0, 14, 64)] = bad
        assert not run(lib, w, one)[0].any()
    nan = np.array(one)
    nan[np.arange(64), 2 * rng.integers(0, 6, 64)] = np.nan
    assert not run(lib, rng.uniform(-1, 1, (64, 14)), nan)[0].any()


def test_link_values(lib):
    v = np.concatenate([[1.0, -1.0, 0.0, np.nan], np.cos(np.linspace(-7, 7, 1001)), 2.0 ** -np.arange(70.0)])
    out = np.empty_like(v)
    lib.h_link(ctypes.c_void_p(v.ctypes.data), ctypes.c_long(v.size), ctypes.c_void_p(out.ctypes.data))
    assert np.array_equal(out[:3], v[:3]) and np.isnan(out[3])
    assert (np.abs(out - v)[4:] <= 2.0 ** -62).all()
