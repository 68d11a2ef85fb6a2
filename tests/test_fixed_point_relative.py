"""The integer Laplacian, current and gradients of the fused FP64 update
(fixed_point.cuh, compiled as host C++) where scalars, components, neighbours or
sines are small beside the others: against long double, in units of the terms
that each result is the sum of.  Within the sum of the truncations (the products
2^-59 of themselves, the alignments one unit each), and on the average no further
off than the same terms by fused multiply-adds in doubles, one rounding per
operation.  On the GPU, whole steps of states with such small parts."""
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
#include <algorithm>
#include <cmath>
using namespace lat;
// u[2], cur[3], grad[6]; scale: the largest term of each
template <class T> static void terms(const T* v, const T* l, T* out, T* scale)
{
    T x[3][2];
    for (int k = 0; k < 2; ++k) scale[k] = std::abs(v[k]);
    for (int a = 0; a < 3; ++a) {
        const T c = l[2 * a], s = l[2 * a + 1], cm = l[6 + 2 * a], sm = l[7 + 2 * a];
        const T* f = v + 2 + 2 * a; const T* b = v + 8 + 2 * a;
        const T A = std::fma(s, f[1], c * f[0]), B = std::fma(-s, f[0], c * f[1]);
        x[a][0] = std::fma(-sm, b[1], std::fma(cm, b[0], A));
        x[a][1] = std::fma(sm, b[0], std::fma(cm, b[1], B));
        out[2 + a] = std::fma(v[1], A, -v[0] * B);
        out[5 + 2 * a] = v[0] - cm * b[0] + sm * b[1];
        out[6 + 2 * a] = v[1] - cm * b[1] - sm * b[0];
        const T tA = std::max(std::abs(c * f[0]), std::abs(s * f[1])), tB = std::max(std::abs(c * f[1]), std::abs(s * f[0]));
        const T t0 = std::max(std::abs(cm * b[0]), std::abs(sm * b[1])), t1 = std::max(std::abs(cm * b[1]), std::abs(sm * b[0]));
        scale[0] = std::max(scale[0], std::max(tA, t0));
        scale[1] = std::max(scale[1], std::max(tB, t1));
        scale[2 + a] = std::max(std::abs(v[1]) * tA, std::abs(v[0]) * tB);
        scale[5 + 2 * a] = std::max(std::abs(v[0]), t0);
        scale[6 + 2 * a] = std::max(std::abs(v[1]), t1);
    }
    for (int k = 0; k < 2; ++k) out[k] = std::fma(T(-6), v[k], x[0][k] + x[1][k] + x[2][k]);
}
// errors in units of the terms, of the integers and of the doubles; the result in those units
extern "C" void h_errors(const double* v, const double* link, long n, double* err, double* derr, double* rel, int* ok)
{
    for (long i = 0; i < n; ++i, v += 14, link += 12, err += 11, derr += 11, rel += 11) {
        double p[2] = {v[0], v[1]}, f[3][2], b[3][2], got[11], g[3][2], cur[3], u[2];
        int64_t cs[3], sn[3], csm[3], snm[3];
        for (int a = 0; a < 3; ++a) {
            for (int k = 0; k < 2; ++k) f[a][k] = v[2 + 2 * a + k], b[a][k] = v[8 + 2 * a + k];
            cs[a] = fix::link_of(link[2 * a]), sn[a] = fix::link_of(link[2 * a + 1]);
            csm[a] = fix::link_of(link[6 + 2 * a]), snm[a] = fix::link_of(link[7 + 2 * a]);
        }
        ok[i] = fix::scalar_terms<true>(p, f, b, cs, sn, csm, snm, u, cur, g);
        for (int k = 0; k < 2; ++k) got[k] = u[k];
        for (int a = 0; a < 3; ++a) got[2 + a] = cur[a], got[5 + 2 * a] = g[a][0], got[6 + 2 * a] = g[a][1];
        double d[11], ds[11];
        terms<double>(v, link, d, ds);
        long double lv[14], ll[12], l[11], s[11];
        for (int k = 0; k < 14; ++k) lv[k] = v[k];
        for (int k = 0; k < 12; ++k) ll[k] = link[k];
        terms<long double>(lv, ll, l, s);
        for (int k = 0; k < 11; ++k) {
            err[k] = (double)((got[k] - l[k]) / s[k]);
            derr[k] = (double)((d[k] - l[k]) / s[k]);
            rel[k] = (double)(l[k] / s[k]);
        }
    }
}
"""

# truncations of a Laplacian, a current and a gradient, in units of their terms
UNITS = np.array([11 * 2.0 ** -57] * 2 + [5.5 * 2.0 ** -58] * 3 + [7 * 2.0 ** -60] * 6)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("relative")
    (d / "drv.cpp").write_text(SRC)
    so = d / "librelative.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CUDA_INC}", f"-I{CSRC}",
                    str(d / "drv.cpp"), "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def errors(lib, v, theta):
    v = np.ascontiguousarray(v.reshape(-1, 14), np.float64)
    link = np.ascontiguousarray(np.stack([np.cos(theta), np.sin(theta)], -1).reshape(-1, 12))
    n = len(v)
    out = [np.zeros((n, 11)) for _ in range(3)]
    ok = np.zeros(n, np.int32)
    P = ctypes.c_void_p
    lib.h_errors(P(v.ctypes.data), P(link.ctypes.data), ctypes.c_long(n), *[P(o.ctypes.data) for o in out], P(ok.ctypes.data))
    return (ok != 0, *out)


def rms(x):
    return np.sqrt(np.mean(x ** 2, 0))


@pytest.mark.parametrize("k", [0, 4, 7, 10, 20, 40])
@pytest.mark.parametrize("small", ["site", "neighbour", "others", "component", "sines", "component and sines"])
def test_small_beside_large(lib, small, k):
    rng = np.random.default_rng(9)
    n = 30000
    ph = rng.uniform(0, 2 * np.pi, (n, 7))
    v = rng.uniform(0.7, 1.3, (n, 7, 1)) * np.stack([np.cos(ph), np.sin(ph)], -1)
    theta = rng.uniform(-0.5, 0.5, (n, 6))
    if small == "site":
        v[:, 0] *= 2.0 ** -k
    elif small == "neighbour":
        v[:, 2] *= 2.0 ** -k
    elif small == "others":      # one neighbour large beside the rest
        v[:, [0, 1, 2, 3, 5, 6]] *= 2.0 ** -k
    if small.startswith("component"):
        v[..., 1] *= 2.0 ** -k
    if small.endswith("sines"):
        theta *= 2.0 ** -k
    ok, err, derr, rel = errors(lib, v, theta)
    assert ok.all()
    assert (np.abs(err) <= UNITS + 2.0 ** -53 * np.abs(rel)).all()
    assert (rms(err) <= rms(derr)).all(), (rms(err) / rms(derr))


@pytest.mark.gpu
@pytest.mark.parametrize("state", ["small component", "small core"])
@pytest.mark.parametrize("diag_every", [0, 1])
def test_steps_keep_small_components(state, diag_every):
    """Nine fused steps on 33x32x34 against the strict form (kernel_variant 1): a
    real scalar whose imaginary part and links are 2^-30 of it, and a region where
    the scalar is 2^-30 of its value elsewhere and the links vanish, each
    component relative to itself, with the bound of the step's other tests."""
    from axions_gb300 import lattice
    from axions_gb300.params import ENERGY_EVOLUTION, F64, F64_FAST, make_params
    sides = (33, 32, 34)
    rng = np.random.default_rng(11)

    def run(ic, precision, variant):
        p = make_params(0, nx=sides[0], ny=sides[1], nz=sides[2], d=0.5, dt=0.05, lam=2.0, g=1.0, alpha=3.0,
                        energy_form=ENERGY_EVOLUTION, precision=precision, kernel_variant=variant)
        with lattice.Lattice(p) as lat:
            lat.set_state(ic, ic, 0)
            lat.advance(9, diag_every=diag_every)
            return lat.get_state()[0].reshape((5,) + sides)

    ic = rng.uniform(0.5, 1.5, (5,) + sides) * rng.choice([-1.0, 1.0], (5,) + sides)
    if state == "small component":
        ic[1:] *= 2.0 ** -30
    else:
        ic[:2, 5:28, 5:28, 5:28] *= 2.0 ** -30
        ic[2:, 4:29, 4:29, 4:29] = 0.0
    want, got = run(ic, F64, 1), run(ic, F64_FAST, 0)
    inner = (slice(None),) * 3 if state == "small component" else (slice(15, 18),) * 3   # nine sites and more from the rest
    for c in range(5):
        w, g = want[c][inner], got[c][inner]
        assert np.linalg.norm(g - w) <= 2e-14 * np.linalg.norm(w), c
