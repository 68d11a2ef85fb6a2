"""The FP32 test that keeps faces out of the double-precision crossing search.

detect_face.cuh is compiled as host C++ (its intrinsics are bit moves; both
builds have contraction off), so the test and the search run here without a
GPU.  A face that face_maybe rejects must have no root in face_roots, for any
corner values: noise, smooth fields down to a gradient of 1e-4 a cell, faces
with a root near an edge or a corner, double roots, a bilinear term that
vanishes exactly or nearly, equal corners, magnitudes from 1e-290 to 1e290,
zeros, Inf and NaN, and lattice positions up to the given distance from the
origin.  The share that is rejected is checked where it has to be large.
"""
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
#define __device__
#define __forceinline__ inline
inline int __double2hiint(double x) { long long u; std::memcpy(&u, &x, 8); return (int)(u >> 32); }
inline int __double2loint(double x) { long long u; std::memcpy(&u, &x, 8); return (int)(unsigned)(u & 0xffffffffLL); }
inline float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
inline unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
using std::fabs; using std::sqrt;
"""

DRIVER = r"""
#include "detect_face.cuh"
// v: [n][4 corners][2], uw: [n][2] integer positions; out: roots, maybe
extern "C" void faces(const double* v, const double* uw, long n, double du, double dw, float eref, int f32, int* roots,
                      int* maybe) {
    for (long i = 0; i < n; ++i) {
        double c[4][2];
        lat::Corner k[4];
        for (int q = 0; q < 4; ++q) {
            for (int m = 0; m < 2; ++m) c[q][m] = f32 ? (double)(float)v[8 * i + 2 * q + m] : v[8 * i + 2 * q + m];
            k[q] = f32 ? lat::Corner{lat::corner_float((float)c[q][0]), lat::corner_float((float)c[q][1])}
                       : lat::Corner{lat::corner_float(c[q][0]), lat::corner_float(c[q][1])};
        }
        roots[i] = lat::face_roots(c[0], c[1], c[2], c[3], uw[2 * i] * du, uw[2 * i + 1] * dw, du, dw).n;
        maybe[i] = lat::face_maybe(k[0], k[1], k[2], k[3], eref);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("face")
    (d / "shim.h").write_text(SHIM)
    (d / "drv.cpp").write_text(DRIVER)
    so = d / "libface.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CUDA_INC}", f"-I{CSRC}",
                    "-include", str(d / "shim.h"), str(d / "drv.cpp"), "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def check(lib, v, half, rng, f32=False, d=(0.5, 0.35)):
    """half: sides/2 of the lattice; returns the share of faces rejected."""
    v = np.ascontiguousarray(v, dtype=np.float64).reshape(-1, 4, 2)
    n = len(v)
    uw = rng.integers(-half, half, (n, 2)).astype(np.float64)
    roots, maybe = np.zeros(n, np.int32), np.zeros(n, np.int32)
    eref = min(1.0, 16 * 2.0 ** -53 * (1.0 + half) ** 3)
    P = ctypes.c_void_p
    lib.faces(P(v.ctypes.data), P(uw.ctypes.data), ctypes.c_long(n), ctypes.c_double(d[0]), ctypes.c_double(d[1]),
              ctypes.c_float(eref), ctypes.c_int(f32), P(roots.ctypes.data), P(maybe.ctypes.data))
    lost = (roots > 0) & (maybe == 0)
    assert not lost.any(), (int(lost.sum()), v[lost][:2].tolist(), uw[lost][:2].tolist())
    return 1 - maybe.mean()


def through(rng, n, grad, second, s, t):
    """Faces whose bilinear interpolants vanish at (s, t): gradients `grad`, bilinear terms `second`."""
    b, c = (rng.normal(size=(n, 2)) * grad for _ in range(2))
    e = rng.normal(size=(n, 2)) * second
    a = -(b * s[:, None] + c * t[:, None] + e * (s * t)[:, None])
    return np.stack([a, a + b, a + c, a + b + c + e], 1)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("half", [4, 64, 512, 2048, 32768])
def test_rejected_faces_have_no_root(lib, half, f32):
    rng = np.random.default_rng(half + f32)
    n = 200_000

    def go(v):
        return check(lib, v, half, rng, f32)

    noise = rng.normal(size=(n, 4, 2))
    share = go(noise)
    if half <= 512:
        assert share > 0.4
    go(np.stack([np.cos(p := rng.uniform(0, 2 * np.pi, (n, 4))), np.sin(p)], -1))
    base = rng.normal(size=(n, 1, 2))
    for grad in (0.3, 0.1, 1e-2, 1e-3, 1e-4):
        b, c = rng.normal(size=(n, 2)) * grad, rng.normal(size=(n, 2)) * grad
        e = rng.normal(size=(n, 2)) * grad ** 2
        share = go(np.stack([base[:, 0], base[:, 0] + b, base[:, 0] + c, base[:, 0] + b + c + e], 1))
        if half <= 512 and grad <= 0.1:
            assert share > 0.8
        # around the zero: inside, at the edges and corners, just outside
        for width in (1.0, 1e-3, 1e-9, 1e-15):
            s = rng.choice([0.0, 0.5, 1.0], n) + rng.normal(size=n) * width
            t = rng.choice([0.0, 0.5, 1.0], n) + rng.normal(size=n) * width
            for second in (grad, grad ** 2, 1e-9 * grad, 0.0):
                go(through(rng, n // 8, grad, second, s[: n // 8], t[: n // 8]))


def test_double_roots_degenerate_and_extreme_faces(lib):
    rng = np.random.default_rng(3)
    n = 100_000
    # v_1 close to a multiple of v_0: the resultant nearly vanishes
    v = rng.normal(size=(n, 4, 2))
    for eps in (1e-2, 1e-5, 1e-8, 1e-12, 0.0):
        w = v.copy()
        w[..., 1] = 0.7 * v[..., 0] + eps * v[..., 1]
        check(lib, w, 256, rng)
    # double roots: v_0 = s - f(t), v_1 touching it
    s0, t0 = rng.uniform(0, 1, n), rng.uniform(0, 1, n)
    st = np.array([[0, 0], [1, 0], [0, 1], [1, 1]], float)
    ds, dt = st[:, 0] - s0[:, None], st[:, 1] - t0[:, None]
    for eps in (0.0, 1e-16, 1e-12, 1e-8, 1e-4, -1e-12, -1e-8, -1e-4):
        v0 = ds + dt
        v1 = ds * dt * rng.normal(size=(n, 1)) + v0 * rng.normal(size=(n, 1)) + eps
        check(lib, np.stack([v0, v1], -1), 256, rng)
    few = rng.integers(-1, 2, (n, 4, 2)).astype(float)   # zeros, equal and opposite corners
    check(lib, few, 256, rng)
    check(lib, few, 256, rng, f32=True)
    for scale in (1e-290, 1e-200, 1e-45, 1e-38, 1e-30, 1e-10, 1e10, 1e30, 1e38, 1e100, 1e200):
        check(lib, scale * rng.normal(size=(n, 4, 2)), 256, rng)
    mixed = rng.normal(size=(n, 4, 2)) * 10.0 ** rng.uniform(-60, 60, (n, 4, 2))
    check(lib, mixed, 256, rng)
    bad = rng.normal(size=(n, 4, 2))
    bad[rng.random(bad.shape) < 0.2] = np.inf
    bad[rng.random(bad.shape) < 0.1] = np.nan
    bad[rng.random(bad.shape) < 0.1] = -np.inf
    check(lib, bad, 256, rng)
