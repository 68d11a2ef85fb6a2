"""The Moore FP64 marching step (moore_march.cuh): the strict form gives bitwise
the fields of the one-pass kernel (kernel_variant 1), which evaluates every
link function where it is used, as the reference does; the fused form
(LAT_F64_FAST) tracks it to the rounding of its operations.  Sides cover tiles
of one and several columns and rows, remainders in y and z, lattices narrower
than a tile, two-site periodic and three-site fixed axes, and x-ranges that end
inside a CTA's chunk; spacings that are powers of two (exact scalings), equal
and unequal, and general ones (quotients)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(sides, d, bc, current, precision=0, variant=0, q=(1.0, 2.0)):
    from axions_gb300.params import ENERGY_EVOLUTION, ENERGY_MPI, MODEL_MOORE, make_params
    nx, ny, nz = sides
    dx, dy, dz = d
    return make_params(MODEL_MOORE, nx=nx, ny=ny, nz=nz, dx=dx, dy=dy, dz=dz, dt=0.2 * min(d), lam=2.0, lambda2=1.5,
                       lambda12=0.3, eta=1.0, eta2=0.9, q1=q[0], q2=q[1], g=0.8, damped_nt=4, dampFac=0.5, alpha=3.0, bc=bc,
                       energy_form=ENERGY_MPI if current else ENERGY_EVOLUTION, moore_current=current,
                       precision=precision, kernel_variant=variant)


@pytest.mark.parametrize("sides,bc", [((2, 2, 2), 0), ((3, 3, 3), 1), ((7, 5, 33), 0), ((6, 130, 3), 0), ((9, 4, 97), 1),
                                      ((20, 21, 64), 0), ((37, 18, 41), 1)])
@pytest.mark.parametrize("d,current,q", [((0.5, 0.5, 0.5), 0, (1.0, 2.0)), ((0.5, 0.25, 1.0), 1, (2.0, 1.0)),
                                         ((0.35, 0.4, 0.3), 1, (1.0, 0.5))])
def test_march_is_bitwise_the_one_pass_step(sides, bc, d, current, q):
    from axions_gb300 import lattice
    from axions_gb300.params import F64_FAST
    ic = lattice.random_phase_ic(_params(sides, d, bc, current, q=q), 5, independent=True)
    ic[4:] = np.random.default_rng(2).uniform(-4, 4, ic[4:].shape)
    res = []
    for precision, variant in ((0, 0), (0, 1), (F64_FAST, 0)):
        with lattice.Lattice(_params(sides, d, bc, current, precision, variant, q)) as lat:
            lat.set_state(ic, ic, 0)
            diags = lat.advance(9, diag_every=3)
            res.append((lat.get_slots(), np.array(diags)))
    assert np.array_equal(res[0][0], res[1][0])
    np.testing.assert_allclose(res[0][1], res[1][1], rtol=1e-12)
    # nine steps of a few hundred roundings each
    assert np.linalg.norm(res[2][0] - res[1][0]) <= 1e-13 * np.linalg.norm(res[1][0])
    np.testing.assert_allclose(res[2][1], res[1][1], rtol=1e-11)
