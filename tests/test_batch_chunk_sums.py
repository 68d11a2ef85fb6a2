"""Diagnostics of batched lattices are the same bits for the default chunk and for
every explicit one that is a multiple of 8, shorter or longer than the x extent,
with x extents that are no multiple of the planes of a partial sum (2, 4 or 8 by the
size).  The scalars span six decades: sums in doubles of single-precision values of
one size would be exact in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(0, (33, 32, 32), 0), (0, (35, 34, 33), 1), (0, (50, 60, 62), 0), (0, (100, 52, 60), 0), (1, (33, 32, 36), 0), (1, (100, 50, 64), 0)]


@pytest.mark.parametrize("model,sides,bc", CASES)
def test_sums_do_not_depend_on_the_chunk(model, sides, bc):
    from axions_gb300 import lattice
    from axions_gb300.params import ENERGY_EVOLUTION, F32, make_params
    nx, ny, nz = sides
    kw = dict(lambda2=0.01, lambda12=0.0, eta2=1.0, q1=1.0, q2=2.0) if model else {}
    p = make_params(model, nx=nx, ny=ny, nz=nz, d=0.5, dt=0.01, lam=0.01, eta=1.0, g=1.0, alpha=3.0, energy_form=ENERGY_EVOLUTION,
                    precision=F32, bc=bc, **kw)
    rng = np.random.default_rng(8)
    ic = np.array(lattice.random_phase_ic(p, 5))
    ic[:-3] *= 10.0 ** rng.uniform(-4, 2, ic.shape[1:])
    ref = None
    for chunk in (0, 8, 64, 128):
        with lattice.Lattice(p) as lat, lattice.Batch(1) as b:
            lat.set_state(ic, ic, 0)
            b.set_chunk(chunk)
            b.add(lat, diag_every=2, stop_step=6)
            b.advance(6)
            out = lat.get_slots(), b.take_diags(lat)
        ref = ref or out
        assert np.array_equal(out[0], ref[0])
        assert out[1] == ref[1], chunk
