"""The FP32 pair step's tiles other than 64x4 with 16-byte staging (Moore
lattices of these shapes take the tiled step): odd sides, fixed z walls, z
extents of one pair, of a partial last pair, of several tiles, 16-byte staged extents such as 32, 48 and 96, rows
narrower than a tile; against the tiled step (kernel_variant 3) and the FP64
path with the bounds of the 64x4 tile's test (other contractions: FP32
accuracy, not bitwise): fields L2 within 2e-6 and max within 2e-5, energies
1e-5 and Gauss sums 1e-4 relative, 12 steps with diagnostics every 4.  A batch
of two such lattices gives the same fields as the lattice in a batch of its
own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [((2, 2, 2), 0, 0), ((3, 3, 3), 1, 0), ((4, 6, 9), 0, 0), ((6, 5, 33), 0, 0), ((9, 4, 97), 1, 0), ((5, 130, 4), 0, 0),
         ((16, 8, 32), 0, 0), ((8, 9, 48), 0, 1), ((7, 12, 96), 1, 1), ((40, 36, 33), 0, 0), ((12, 21, 83), 1, 0),
         ((6, 7, 66), 0, 2), ((33, 31, 130), 0, 0)]


def _params(model, sides, bc, bc_z, **kw):
    from axions_gb300.params import ENERGY_EVOLUTION, MODEL_MOORE, make_params
    nx, ny, nz = sides
    base = dict(nx=nx, ny=ny, nz=nz, d=0.5, dt=0.1, lam=2.0, eta=1.0, g=0.8, damped_nt=3, dampFac=0.5, alpha=3.0, bc=bc,
                bc_z=bc_z, energy_form=ENERGY_EVOLUTION)
    if model:
        base.update(lambda2=2.0, lambda12=0.3, eta2=1.0, q1=1.0, q2=2.0 if model == 1 else -1.0, moore_current=1)
    base.update(kw)
    return make_params(MODEL_MOORE if model else 0, **base)


def normwise(a, b):
    d = np.abs(a - b)
    return d.max() / np.abs(b).max(), np.linalg.norm(d) / np.linalg.norm(b)


@pytest.mark.parametrize("model", [0, 1, 2])   # 2: Moore with charges other than (1, 2)
@pytest.mark.parametrize("sides,bc,bc_z", SIDES)
def test_pair_shapes_tracks_tiled_and_fp64(model, sides, bc, bc_z):
    from axions_gb300 import lattice
    from axions_gb300.params import F32
    if bc_z == 2 and sides[2] < 3:
        pytest.skip("fixed axes need three sites")
    p = _params(model, sides, bc, bc_z)
    ic = lattice.random_phase_ic(p, 41, independent=model > 0)
    res = {}
    for name, prec, var in (("f64", 0, 0), ("pair", F32, 0), ("tiled", F32, 3)):
        q = p.copy()
        q.precision, q.kernel_variant = prec, var
        with lattice.Lattice(q) as lat:
            lat.set_state(ic, ic, 0)
            d = lat.advance(12, diag_every=4)
            res[name] = (lat.get_slots(), d)
    s64, d64 = res["f64"]
    for name in ("pair", "tiled"):
        st, d = res[name]
        mx, l2 = normwise(st, s64)
        assert l2 < 2e-6 and mx < 2e-5, (name, mx, l2)
        np.testing.assert_allclose([x[1] for x in d], [x[1] for x in d64], rtol=1e-5)
        np.testing.assert_allclose([x[2] for x in d], [x[2] for x in d64], rtol=1e-4)
    assert normwise(res["pair"][0], res["tiled"][0])[1] < 2e-6


def test_pair_shapes_in_a_batch_alone_and_with_others():
    from axions_gb300 import lattice
    from axions_gb300.params import F32

    def run(specs):
        lats = []
        for model, sides, bc, bc_z in specs:
            p = _params(model, sides, bc, bc_z, precision=F32)
            lat = lattice.Lattice(p)
            ic = lattice.random_phase_ic(p, 7, independent=model > 0)
            lat.set_state(ic, ic, 0)
            lats.append(lat)
        with lattice.Batch(8) as b:
            for lat in lats:
                b.add(lat, diag_every=3, stop_step=11)
            while b.advance(4) > 0:
                pass
            out = [(lat.get_slots(), b.take_diags(lat)) for lat in lats]
        for lat in lats:
            lat.close()
        return out

    specs = [(m, s, bc, bz) for m, (s, bc, bz) in zip((0, 1, 2, 0, 1, 2), SIDES[3:9])]
    mix = run(specs)
    for spec, (st, d) in zip(specs, mix):
        [(st1, d1)] = run([spec])
        assert np.array_equal(st, st1) and d == d1
