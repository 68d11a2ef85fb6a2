"""Workloads of the lattice framework, as its users run them, for timing and for comparing results.

Every case goes through the public entry points (the Python mirror of the C ABI, `axions_gb300.lattice`, and for
caller-owned fields the C entry itself).  The kinds:

  caller     lat_ah_step_f64_noalloc on fields the caller owns on the device: a solver loop with its own memory
  run64      one whole FP64 run from host state to host state (Lattice.run): upload, steps, diagnostics, download
  run32      one FP32 run: device-drawn initial state, steps with diagnostics, the final level dumped by a snapshot
  crossings  the list of string crossings of a level in the caller's buffer (lat_detect_crossings)
  strings    total string length and plaquette winding of a level (Lattice.string_length, Lattice.winding)
  ensemble   independent FP32 lattices advanced together (Batch), diagnostics and final levels read back

An FP32 lattice's level and its diagnostics are handed on in float32: the lattice holds no more than that.

`listed()` gives the fixed cases, `draw(rng)` more of the same ranges, `prepare`/`run` the inputs and one pass,
`work` the bytes and operations a pass cannot do without, `exact` the same results in plain 64-bit torch or numpy.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from axions_gb300 import lattice
from axions_gb300.params import ENERGY_EVOLUTION, F32, F64, F64_FAST, MODEL_AH, MODEL_MOORE, make_params

PRECISION = {"f32": F32, "f64": F64, "f64_fast": F64_FAST}
BC = {"periodic": 0, "fixed": 1}


def _case(name, kind, n, **kw):
    """A case with every key of its kind; `n` is (nx, ny, nz)."""
    c = {"name": name, "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "model": "ah", "precision": "f64", "walls": "periodic",
         "spacing": 0.5, "dt": 0.1, "lam": 2.0, "g": 1.0, "alpha": 3.0, "damped": 0, "steps": 1, "diag_every": 0,
         "pinned": False, "q1": 1.0, "q2": 2.0, "jobs": 1, "tick": 25, "modes": 0}
    unknown = set(kw) - set(c)
    if unknown:
        raise KeyError(unknown)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest calls: a host solver stepping a small box it owns, a few steps per call
        _case("caller_24", "caller", (24, 24, 24), steps=4),
        # one member of an ensemble of small lattices, stepped on its own
        _case("ah32_small", "run32", (40, 36, 33), precision="f32", steps=200, diag_every=20),
        # the plain FP64 configuration: 128^3, Minkowski, energy and Gauss every 10 steps, arrays from ordinary memory
        _case("ah64_128", "run64", (128, 128, 128), alpha=0.0, steps=50, diag_every=10),
        # the fused FP64 form on a large periodic box, radiation era, pinned buffers; the largest case
        _case("ah64fast_384", "run64", (384, 384, 384), precision="f64_fast", steps=10, diag_every=20, pinned=True),
        # evolution's loop: fixed walls, an odd box with a general spacing, damping, energy and Gauss at every step
        _case("ah64_walls", "run64", (101, 99, 97), walls="fixed", spacing=0.35, dt=0.07, damped=15, steps=30, diag_every=1),
        # the two-scalar model in FP64
        _case("moore64_96", "run64", (96, 96, 96), model="moore", steps=40, diag_every=20, pinned=True),
        # the FP32 form on a box of the serving and production sizes
        _case("ah32_256", "run32", (256, 256, 256), precision="f32", steps=300, diag_every=20),
        # the reference programs' own sides are odd (1001, 401); fixed walls as evolution has them
        _case("ah32_odd", "run32", (201, 199, 203), precision="f32", walls="fixed", spacing=0.25, dt=0.05, lam=1.0, damped=100,
              steps=150, diag_every=25),
        # the two-scalar model in FP32, charges 1 and 2, radiation era
        _case("moore32_192", "run32", (192, 192, 192), model="moore", precision="f32", steps=200, diag_every=20),
        # crossings of a noisy level (about one per site, as gauged runs have after a few hundred steps)
        _case("crossings_noise", "crossings", (96, 100, 104)),
        # length and winding of a string network in a large FP32 box
        _case("strings_256", "strings", (256, 256, 256), precision="f32", g=0.0, spacing=0.25, dt=0.05, lam=1.0, modes=6),
        # an ensemble of small lattices, mixed couplings, both models
        _case("ensemble_64", "ensemble", (64, 64, 64), precision="f32", jobs=24, steps=100, tick=25, diag_every=20),
    ]


def _side(rng, lo, hi):
    """A side between lo and hi, spread over the logarithm; one in three odd or otherwise ragged."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.67:
        v = max(8, (v + 2) // 4 * 4)
    return min(max(v, lo), hi)


def _box(rng, lo, hi):
    if rng.random() < 0.5:
        n = _side(rng, lo, hi)
        return (n, n, n)
    n = _side(rng, lo, hi)
    return tuple(min(hi, max(lo, int(n * rng.uniform(0.75, 1.25)) if rng.random() < 0.5 else n)) for _ in range(3))


def draw(rng):
    kind = rng.choice(["caller", "run64", "run64", "run64", "run32", "run32", "run32", "crossings", "strings", "ensemble"])
    lam, g = round(rng.uniform(0.5, 4.0), 4), round(rng.uniform(0.5, 1.5), 4)
    spacing, dt = rng.choice([(0.5, 0.1), (0.25, 0.05), (0.35, 0.07)])
    common = {"lam": lam, "g": g, "spacing": spacing, "dt": dt, "alpha": rng.choice([0.0, 3.0])}
    walls = rng.choice(["periodic", "periodic", "fixed"])
    if kind == "caller":
        n = _box(rng, 12, 60)
        c = _case("", kind, n, precision=rng.choice(["f64", "f64_fast"]), walls=walls, damped=rng.choice([0, 3]),
                  steps=rng.randint(1, 12), **common)
    elif kind == "run64":
        model = rng.choice(["ah", "ah", "moore"])
        n = _box(rng, 40, 256 if model == "ah" else 128)
        sites = n[0] * n[1] * n[2]
        steps = max(4, min(60, int(1.2e8 / sites)))
        c = _case("", kind, n, model=model, precision=rng.choice(["f64", "f64_fast"]), walls=walls, damped=rng.choice([0, steps // 2]),
                  steps=steps, diag_every=rng.choice([1, 5, 10, 20]), pinned=rng.random() < 0.5, **common)
    elif kind == "run32":
        model = rng.choice(["ah", "ah", "moore"])
        n = _box(rng, 32, 256 if model == "ah" else 208)
        sites = n[0] * n[1] * n[2]
        q = rng.choice([(1.0, 2.0), (2.0, 1.0), (1.0, 2.0)])
        c = _case("", kind, n, model=model, precision="f32", walls=walls, q1=q[0], q2=q[1], damped=rng.choice([0, 20]),
                  steps=max(30, min(120, int(8e8 / sites))), diag_every=rng.choice([5, 10, 20]), **common)
    elif kind == "crossings":
        c = _case("", kind, _box(rng, 32, 128), precision=rng.choice(["f64", "f32"]), walls=walls, modes=rng.choice([0, 0, 5, 10]), **common)
    elif kind == "strings":
        n = _side(rng, 64, 256)
        c = _case("", kind, (n, n, n), precision=rng.choice(["f64", "f32"]), modes=rng.randint(3, 6), **common)
    else:
        n = _side(rng, 32, 96)
        jobs = rng.randint(4, 24)
        steps = max(25, min(100, int(1.0e9 / (n ** 3 * jobs))))
        c = _case("", kind, (n, n, n), precision="f32", jobs=jobs, steps=steps, tick=rng.choice([25, 50]),
                  diag_every=rng.choice([10, 20]), **common)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _params(c, lam=None, g=None, model=None):
    moore = (model or c["model"]) == "moore"
    kw = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], d=c["spacing"], dt=c["dt"], lam=c["lam"] if lam is None else lam, eta=1.0,
              g=c["g"] if g is None else g, damped_nt=c["damped"], dampFac=0.5 if c["damped"] else 0.0, alpha=c["alpha"], scaling=1.0,
              tau0=1.0, energy_form=ENERGY_EVOLUTION, precision=PRECISION[c["precision"]], bc=BC[c["walls"]])
    if moore:
        return make_params(MODEL_MOORE, lambda2=kw["lam"], lambda12=0.0, eta2=1.0, q1=c["q1"], q2=c["q2"], **kw)
    return make_params(MODEL_AH, **kw)


def _ensemble(c, seed):
    """(params, seed of the initial state) of every lattice: its own couplings, one in four a Moore lattice."""
    r = np.random.default_rng(seed)
    return [(_params(c, lam=float(r.uniform(0.5, 4.0)), g=float(r.uniform(0.5, 1.5)), model="moore" if q % 4 == 3 else "ah"),
             int(r.integers(1 << 40))) for q in range(c["jobs"])]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _level(c, seed):
    """A starting level as the reference's programs draw it: uniform phases, |phi| = 1, no gauge field."""
    gen = _generator(seed)
    shape = (c["nx"], c["ny"], c["nz"])
    out = []
    for _ in range(2 if c["model"] == "moore" else 1):
        ph = 2 * math.pi * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
        out += [torch.cos(ph), torch.sin(ph)]
    out += [torch.zeros(shape, device="cuda", dtype=torch.float64) for _ in range(3)]
    return out


def _scalar(c, seed):
    """A level's scalar for detection: modes == 0 uncorrelated phases and magnitudes; else a smooth Gaussian field
    (wavenumbers up to `modes` per side), whose zeros are a network of strings."""
    gen = _generator(seed)
    shape = (c["nx"], c["ny"], c["nz"])
    if c["modes"] == 0:
        ph = 2 * math.pi * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
        mag = 0.5 + torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
        return [mag * torch.cos(ph), mag * torch.sin(ph)]
    m = c["modes"]
    amp = torch.randn((2 * m + 1,) * 3 + (2,), generator=gen, device="cuda", dtype=torch.float64)
    spec = torch.zeros(shape, device="cuda", dtype=torch.complex128)
    k = [torch.arange(-m, m + 1, device="cuda") % n for n in shape]
    spec[k[0][:, None, None], k[1][None, :, None], k[2][None, None, :]] = torch.view_as_complex(amp)
    f = torch.fft.ifftn(spec) * spec.numel() / (2 * m + 1) ** 1.5
    return [f.real.contiguous(), f.imag.contiguous()]


def _host(fields, array):
    """The fields, one after another, in a host array [fields][sites]."""
    t = torch.from_numpy(array)
    for q, f in enumerate(fields):
        t[q].copy_(f.reshape(-1))
    return array


def _buffer(pinned, shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=bool(pinned)).numpy()


def prepare(case, seed):
    c = case
    kind = c["kind"]
    s = {"case": c, "seed": int(seed)}
    if kind == "caller":
        p = _params(c)
        lev = torch.stack(_level(c, seed)).reshape(p.ncomp, 1, p.N)
        s["params"] = p
        s["initial"] = lev.expand(p.ncomp, 2, p.N).contiguous()   # both levels: a stationary start
        s["fields"] = torch.empty_like(s["initial"])
        s["library"] = lattice.load_library()
    elif kind == "run64":
        p = _params(c)
        s["lat"] = lattice.Lattice(p)
        s["now"] = _host(_level(c, seed), _buffer(c["pinned"], (p.ncomp, p.N)))
        s["out"] = _buffer(c["pinned"], (p.ncomp, p.N))
    elif kind == "run32":
        p = _params(c)
        s["lat"] = lattice.Lattice(p)
        s["dump"] = _buffer(True, (p.ncomp, p.N))
        s["level"] = torch.empty((p.ncomp, p.N), dtype=torch.float32)
    elif kind in ("crossings", "strings"):
        p = _params(c)
        s["lat"] = lattice.Lattice(p)
        now = np.zeros((p.ncomp, p.N))
        _host(_scalar(c, seed), now)
        s["lat"].set_state(now)
        if kind == "crossings":
            # room for the crossings of any level of this size; what lies beyond the count stays zero
            s["list"] = _buffer(c["pinned"], (2 * p.N, 3))
            s["list"][:] = 0.0
            s["count"] = ctypes.c_int64(0)
    elif kind == "ensemble":
        s["jobs"] = _ensemble(c, seed)
        s["lats"] = [lattice.Lattice(p) for p, _ in s["jobs"]]
        s["dump"] = [_buffer(True, (p.ncomp, p.N)) for p, _ in s["jobs"]]
        s["level"] = [torch.empty((p.ncomp, p.N), dtype=torch.float32) for p, _ in s["jobs"]]
        s["batch"] = lattice.Batch(max(4, c["jobs"]))
    else:
        raise KeyError(kind)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "caller":
        s["fields"].copy_(s["initial"])
        rc = s["library"].lat_ah_step_f64_noalloc(ctypes.byref(s["params"]), ctypes.c_void_p(s["fields"].data_ptr()), 0, c["steps"],
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(s["library"].lat_last_error())
        return s["fields"]
    lat = s.get("lat")
    if kind == "run64":
        diags, now, _ = lat.run(s["now"], None, 0, c["steps"], c["diag_every"], now_out=s["out"], past_level=False)
        return {"level": now, "diagnostics": np.asarray(diags, dtype=np.float64).reshape(-1, 3)}
    if kind == "run32":
        lat.random_phase_ic_device(s["seed"], independent=True)
        diags = lat.advance(c["steps"], c["diag_every"])
        lat.snapshot_begin(lattice.SNAP_LEVEL, s["dump"])
        lat.snapshot_wait()
        s["level"].copy_(torch.from_numpy(s["dump"]))
        return {"level": s["level"], "diagnostics": np.asarray(diags, dtype=np.float32).reshape(-1, 3)}
    if kind == "crossings":
        rc = lat.L.lat_detect_crossings(lat.h, 0, s["list"].ctypes.data_as(ctypes.POINTER(ctypes.c_double)), len(s["list"]), ctypes.byref(s["count"]))
        if rc:
            raise RuntimeError(lat.L.lat_last_error())
        return {"crossings": s["list"], "count": s["count"].value}
    if kind == "strings":
        l0, l1, count = lat.string_length(0)
        _, winding = lat.winding(0, want_array=False)
        return {"length": [l0, l1], "crossings": count, "winding": winding}
    lats, batch = s["lats"], s["batch"]
    for one, (_, seed) in zip(lats, s["jobs"]):
        one.random_phase_ic_device(seed, independent=True)
        batch.add(one, diag_every=c["diag_every"], stop_step=c["steps"])
    while batch.advance(c["tick"]):
        pass
    diags = []
    for one, dump in zip(lats, s["dump"]):
        one.snapshot_begin(lattice.SNAP_LEVEL, dump)
        diags.append(np.asarray(batch.take_diags(one), dtype=np.float32).reshape(-1, 3))
        batch.remove(one)
    for one, dump, level in zip(lats, s["dump"], s["level"]):
        one.snapshot_wait()
        level.copy_(torch.from_numpy(dump))
    return {"levels": s["level"], "diagnostics": diags}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c = case
    n = c["nx"] * c["ny"] * c["nz"]
    elem = 4 if c["precision"] == "f32" else 8

    def steps(ncomp):
        # per site and step: the two levels read, the next written; the operations of the update, three sincos of
        # the links and the plaquette sines among them (about 20 operations a function)
        return n * c["steps"] * 3 * ncomp * elem, n * c["steps"] * (300 if ncomp == 5 else 480)

    ncomp = 7 if c["model"] == "moore" else 5
    if c["kind"] == "caller":
        b, f = steps(ncomp)
    elif c["kind"] == "run64":
        b, f = steps(ncomp)
        b += 2 * ncomp * n * 8          # the level in, the level out
    elif c["kind"] == "run32":
        b, f = steps(ncomp)
        b += 2 * 2 * ncomp * n * 4 + ncomp * n * 8
    elif c["kind"] == "crossings":
        b, f = 2 * n * elem + (24 * n if c["modes"] == 0 else 0), 3 * 60 * n
    elif c["kind"] == "strings":
        b, f = 2 * 2 * n * elem, (3 * 60 + 3 * 4 * 3) * n
    else:
        a, m = steps(5), steps(7)
        moore = c["jobs"] // 4
        b = (c["jobs"] - moore) * a[0] + moore * m[0] + n * 8 * (5 * (c["jobs"] - moore) + 7 * moore)
        f = (c["jobs"] - moore) * a[1] + moore * m[1]
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit arithmetic
# ---------------------------------------------------------------------------
def _philox(n, seed):
    """Outputs 0..3 of Philox-4x32-10 for counters (s, 0, 0, 0) and the seed as key."""
    mask = 0xFFFFFFFF
    ctr = [torch.arange(n, device="cuda", dtype=torch.int64)] + [torch.zeros(n, device="cuda", dtype=torch.int64) for _ in range(3)]
    k0, k1 = seed & mask, (seed >> 32) & mask

    def mul(a, m):
        lo = (a & 0xFFFF) * m
        mid = (a >> 16) * m + (lo >> 16)
        return mid >> 16, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)

    for r in range(10):
        hi0, lo0 = mul(ctr[0], 0xD2511F53)
        hi1, lo1 = mul(ctr[2], 0xCD9E8D57)
        ctr = [hi1 ^ ctr[1] ^ k0, lo1, hi0 ^ ctr[3] ^ k1, lo0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return ctr


def _device_phases(shape, moore, seed):
    """The device-drawn start of a float32 lattice: its scalars as float32 holds them."""
    n = shape[0] * shape[1] * shape[2]
    w = _philox(n, seed)
    out = []
    for a, b in ((w[0], w[1]), (w[2], w[3]))[: 2 if moore else 1]:
        ph = (2.0 * math.pi) * (((a >> 5) * (1 << 26) + (b >> 6)).double() * (1.0 / 9007199254740992.0))
        out += [torch.cos(ph).float().double().reshape(shape), torch.sin(ph).float().double().reshape(shape)]
    return out + [torch.zeros(shape, device="cuda", dtype=torch.float64) for _ in range(3)]


def _evolve(p, level, steps, diag_every):
    """The leapfrog of the Abelian-Higgs or Moore model from a stationary start; returns (last level, diagnostics)."""
    moore = p.model == MODEL_MOORE
    ns = 2 if moore else 1
    q = [p.q1, p.q2] if moore else [1.0]
    lam, eta2 = [p.lam, p.lambda2], [p.eta ** 2, p.eta2 ** 2]
    d, dt = [p.dx, p.dy, p.dz], p.dt
    phi = [torch.complex(level[2 * a], level[2 * a + 1]) for a in range(ns)]
    th = level[2 * ns:]
    phi_old, th_old = [f.clone() for f in phi], [t.clone() for t in th]
    inner = (slice(1, -1),) * 3 if p.bc else (slice(None),) * 3

    def fwd(f, m):
        return torch.roll(f, -1, m)

    def back(f, m):
        return torch.roll(f, 1, m)

    def div(t):
        return sum((t[m] - back(t[m], m)) / d[m] ** 2 for m in range(3))

    said = []
    for n in range(steps):
        damp = p.dampFac if n < p.damped_nt else 0.0
        fric = damp + p.alpha * p.scaling / (p.tau0 + n * dt)
        diag = diag_every > 0 and n % diag_every == 0
        mag = [f.real ** 2 + f.imag ** 2 - eta2[a] for a, f in enumerate(phi)]
        cur = [0.0, 0.0, 0.0]
        new = []
        grad = 0.0
        for a in range(ns):
            pot = 0.5 * lam[a] * mag[a]
            if moore:
                pot = pot + 0.5 * p.lambda12 * mag[1 - a]
            acc = -pot * phi[a]
            for m in range(3):
                u = torch.polar(torch.ones_like(th[m]), q[a] * th[m])
                ahead = torch.conj(u) * fwd(phi[a], m)
                behind = back(u * phi[a], m)
                acc = acc + (ahead + behind - 2 * phi[a]) / d[m] ** 2
                cur[m] = cur[m] + (phi[a] * torch.conj(ahead)).imag
                if diag:
                    g = (phi[a] - behind) / d[m]
                    grad = grad + g.real ** 2 + g.imag ** 2
                del u, ahead, behind
            acc = acc - fric * (phi[a] - phi_old[a]) / dt
            new.append(2 * phi[a] - phi_old[a] + dt ** 2 * acc)
            del acc
        plaq = {(m, r): th[m] + fwd(th[r], m) - fwd(th[m], r) - th[r] for m, r in ((0, 1), (0, 2), (1, 2))}
        sine = {k: torch.sin(v) for k, v in plaq.items()}
        new_th = []
        for m in range(3):
            acc = -2 * p.g * p.g * cur[m]
            for r in range(3):
                if r != m:
                    f = sine[(m, r)] if m < r else -sine[(r, m)]
                    acc = acc - (f - back(f, r)) / d[r] ** 2
            if damp:
                acc = acc - damp * (th[m] - th_old[m]) / dt
            new_th.append(2 * th[m] - th_old[m] + dt ** 2 * acc)
        if diag:
            vel = [(f - o) / dt for f, o in zip(phi, phi_old)]
            e = grad + sum(v.real ** 2 + v.imag ** 2 for v in vel) + sum(0.25 * lam[a] * mag[a] ** 2 for a in range(ns))
            if moore:
                e = e + 0.5 * p.lambda12 * mag[0] * mag[1]
            gauss = torch.zeros_like(mag[0])
            if p.g != 0:
                e = e + 0.5 * sum(((th[m] - th_old[m]) / (p.g * dt * d[m])) ** 2 for m in range(3))
                e = e + sum(2 * torch.sin(0.5 * v) ** 2 / (p.g * d[m] * d[r]) ** 2 for (m, r), v in plaq.items())
                gauss = (div(th) - div(th_old)) / dt / p.g
                for a in range(ns):
                    gauss = gauss - 2 * p.g * q[a] * (phi[a].imag * vel[a].real - phi[a].real * vel[a].imag)
            said.append([float(n), float((e[inner] * (p.dx * p.dy * p.dz)).sum()), float(gauss[inner].abs().sum())])
        for old, now, nxt in list(zip(phi_old, phi, new)) + list(zip(th_old, th, new_th)):
            if p.bc:
                old_new = now.clone()
                old[inner] = nxt[inner]       # the outer layer of each slot stays as it was given
                now.copy_(old)
                old.copy_(old_new)
            else:
                old.copy_(now)
                now.copy_(nxt)
    out = []
    for f in phi:
        out += [f.real, f.imag]
    out += list(th)
    return torch.stack([f.reshape(-1) for f in out]), np.asarray(said, dtype=np.float64).reshape(-1, 3)


def _crossings(c, re, im):
    """Bilinear zero crossings of every positive face, in the order of the sites."""
    n = [c["nx"], c["ny"], c["nz"]]
    d = c["spacing"]
    v = [re, im]
    x = [((torch.arange(n[m], device="cuda") - int(0.5 * (n[m] - 1))).double() * d).reshape([-1 if r == m else 1 for r in range(3)]).expand(n)
         for m in range(3)]
    rows, valid = [], []
    for a, b in ((0, 1), (0, 2), (1, 2)):    # faces along z, y, x
        u, w = x[a], x[b]
        co = []
        for f in v:
            v00, v10, v01 = f, torch.roll(f, -1, a), torch.roll(f, -1, b)
            v11 = torch.roll(v10, -1, b)
            co.append((v11 - v10 - v01 + v00, (w + d) * (v10 - v00) + w * (v01 - v11), (u + d) * (v01 - v00) + u * (v10 - v11),
                       (u + d) * ((w + d) * v00 - w * v01) - u * ((w + d) * v10 - w * v11)))
        (p1, p2, p3, p4), (q1, q2, q3, q4) = co
        aa = q1 * p3 - p1 * q3
        bb = q1 * p4 + q2 * p3 - p1 * q4 - p2 * q3
        cc = q2 * p4 - p2 * q4
        disc = bb * bb - 4 * aa * cc
        root = torch.sqrt(torch.clamp(disc, min=0))
        lin = aa == 0
        for sign in (1, -1):
            t = (-bb + root) / (2 * aa) if sign > 0 else (-bb - root) / (2 * aa)
            ok = ~lin & (disc >= 0)
            if sign > 0:
                t = torch.where(lin, -cc / bb, t)
                ok = ok | (lin & (bb != 0))
            r = -(p3 * t + p4) / (p1 * t + p2)
            valid.append(ok & (t >= w) & (t <= w + d) & (r >= u) & (r <= u + d))
            rows.append(torch.stack([r if m == a else t if m == b else x[m] for m in range(3)], -1))
    if c["walls"] == "fixed":
        inside = torch.zeros(n, dtype=torch.bool, device="cuda")
        inside[1:-1, 1:-1, 1:-1] = True
        valid = [ok & inside for ok in valid]
    return torch.stack(rows, 3)[torch.stack(valid, 3)].cpu().numpy()


def _length(c, xyz):
    """Greedy chaining of the crossings of a periodic box: (inside the central box, outside)."""
    n, d = [c["nx"], c["ny"], c["nz"]], c["spacing"]
    box = [m * d for m in n]
    cut = (d * d + d * d + d * d) ** 2
    cells = [max(1, int(b / (1.001 * math.sqrt(cut)))) for b in box]
    at = [[min(int((float(p[m]) + int(0.5 * (n[m] - 1)) * d) / box[m] * cells[m]), cells[m] - 1) for m in range(3)] for p in xyz]
    grid = {}
    for j, a in enumerate(at):
        grid.setdefault(tuple(a), []).append(j)
    pts = [tuple(float(t) for t in p) for p in xyz]

    def dist2(p, q):
        s = 0.0
        for m in range(3):
            t = abs(p[m] - q[m])
            t = p[m] - q[m] if t <= 0.5 * box[m] else box[m] - t
            s += t * t
        return s

    alive, total = [True] * len(pts), [0.0, 0.0]
    f = first = 0
    begin = pts[0] if pts else None
    for _ in range(len(pts)):
        best, took = cut, -1
        for i in {(at[f][0] + o) % cells[0] for o in (-1, 0, 1)}:
            for j in {(at[f][1] + o) % cells[1] for o in (-1, 0, 1)}:
                for k in {(at[f][2] + o) % cells[2] for o in (-1, 0, 1)}:
                    for m in grid.get((i, j, k), ()):
                        if alive[m] and m != f:
                            s = dist2(pts[f], pts[m])
                            if s < best or (s == best and m > took):
                                best, took = s, m
        part = 0 if all(-0.25 * box[m] <= pts[f][m] <= 0.25 * box[m] for m in range(3)) else 1
        alive[f] = False
        if took >= 0:
            total[part] += math.sqrt(best)
            f = took
            continue
        if dist2(pts[f], begin) <= cut:
            total[part] += math.sqrt(cut)
        while first < len(pts) and not alive[first]:
            first += 1
        if first < len(pts):
            f, begin = first, pts[first]
    return total


def _winding(re, im):
    """Sum of |winding| over all faces of a periodic box."""
    ph = torch.atan2(im, re)
    total = 0
    for a, b in ((0, 1), (0, 2), (1, 2)):
        loop = [ph, torch.roll(ph, -1, a), torch.roll(torch.roll(ph, -1, a), -1, b), torch.roll(ph, -1, b)]
        s = 0.0
        for e in range(4):
            t = loop[(e + 1) % 4] - loop[e]
            s = s + t - 2 * math.pi * torch.round(t / (2 * math.pi))
        total += int(torch.round(s / (2 * math.pi)).abs().sum())
    return total


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "caller":
        p = _params(c)
        last, _ = _evolve(p, _level(c, seed), c["steps"], 0)
        before, _ = _evolve(p, _level(c, seed), c["steps"] - 1, 0)
        slots = [None, None]
        slots[(c["steps"] + 1) % 2], slots[c["steps"] % 2] = last, before
        return torch.stack(slots, 1)
    if kind == "run64":
        level, said = _evolve(_params(c), _level(c, seed), c["steps"], c["diag_every"])
        return {"level": level, "diagnostics": said}
    if kind == "run32":
        start = _device_phases((c["nx"], c["ny"], c["nz"]), c["model"] == "moore", int(seed))
        level, said = _evolve(_params(c), start, c["steps"], c["diag_every"])
        return {"level": level, "diagnostics": said}
    if kind in ("crossings", "strings"):
        re, im = _scalar(c, seed)
        if c["precision"] == "f32":
            re, im = re.float().double(), im.float().double()
        xyz = _crossings(c, re, im)
        if kind == "crossings":
            full = np.zeros((2 * c["nx"] * c["ny"] * c["nz"], 3))
            full[:len(xyz)] = xyz
            return {"crossings": full, "count": len(xyz)}
        return {"length": [float(t) for t in _length(c, xyz)], "crossings": len(xyz), "winding": _winding(re, im)}
    levels, diags = [], []
    for p, s in _ensemble(c, seed):
        start = _device_phases((c["nx"], c["ny"], c["nz"]), p.model == MODEL_MOORE, s)
        level, said = _evolve(p, start, c["steps"], c["diag_every"])
        levels.append(level)
        diags.append(said)
    return {"levels": levels, "diagnostics": diags}
