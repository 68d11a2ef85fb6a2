"""The strict FP64 Abelian-Higgs update with products by integer instructions
(ah_twopass.cuh) gives bitwise the fields of the one-pass kernel
(kernel_variant 1): lattices on both sides of the size from which it is taken,
spacings with exact scalings and general ones, and states that leave the
integer product's range at some sites only: vanishing link phases (zero sines),
zero scalars, scalars whose products are subnormal, and large ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides,bc", [((31, 32, 33), 0), ((32, 32, 32), 0), ((33, 41, 29), 1)])
@pytest.mark.parametrize("d", [(0.5, 0.5, 0.5), (0.5, 0.25, 1.0), (0.35, 0.4, 0.3)])
@pytest.mark.parametrize("state", ["plain", "edges"])
def test_integer_products_are_bitwise_the_one_pass_step(sides, bc, d, state):
    from axions_gb300 import lattice
    from axions_gb300.params import ENERGY_EVOLUTION, make_params
    nx, ny, nz = sides

    def params(variant):
        return make_params(0, nx=nx, ny=ny, nz=nz, dx=d[0], dy=d[1], dz=d[2], dt=0.05, lam=2.0, g=1.0, damped_nt=4,
                           dampFac=0.5, alpha=3.0, bc=bc, energy_form=ENERGY_EVOLUTION, kernel_variant=variant)

    rng = np.random.default_rng(8)
    ic = np.array(lattice.random_phase_ic(params(0), 5))
    ic[2:] = rng.uniform(-4, 4, ic[2:].shape)
    if state == "edges":
        pick = rng.random(ic.shape[1:])
        ic[2:, pick < 0.1] = 0.0
        ic[:2, (pick > 0.1) & (pick < 0.12)] = 0.0
        ic[:2, (pick > 0.2) & (pick < 0.3)] *= 2.0 ** rng.integers(-1070, -490, 1)[0]
        ic[:2, (pick > 0.3) & (pick < 0.31)] *= 1e-155
        ic[:2, (pick > 0.4) & (pick < 0.401)] *= 30.0
    res = []
    for variant in (0, 1):
        with lattice.Lattice(params(variant)) as lat:
            lat.set_state(ic, ic, 0)
            diags = lat.advance(5, diag_every=2)
            res.append((lat.get_slots(), diags))
    assert np.isfinite(res[1][0]).all()
    assert np.array_equal(res[0][0], res[1][0])
    assert res[0][1] == res[1][1]
