"""The fused FP64 Abelian-Higgs step on both sides of the size from which its
Laplacian and current are in fixed point (ah_twopass.cuh), against the strict
form (kernel_variant 1): random and edge states (zero and tiny scalars at some
sites, no gauge field), walls, friction; and a state with an infinite value
spreads as in the FP64 form: what is not finite there is not finite here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(sides, bc, d, precision, variant=0):
    from axions_gb300.params import ENERGY_EVOLUTION, make_params
    nx, ny, nz = sides
    return make_params(0, nx=nx, ny=ny, nz=nz, dx=d, dy=d, dz=d, dt=0.05, lam=2.0, g=1.0, damped_nt=4, dampFac=0.5, alpha=3.0,
                       bc=bc, energy_form=ENERGY_EVOLUTION, precision=precision, kernel_variant=variant)


def _run(lattice, p, ic, steps=9):
    with lattice.Lattice(p) as lat:
        lat.set_state(ic, ic, 0)
        diags = np.array(lat.advance(steps, diag_every=4))
        return lat.get_slots(), diags


@pytest.mark.parametrize("sides,bc", [((31, 32, 33), 0), ((32, 32, 32), 0), ((41, 37, 33), 1)])
@pytest.mark.parametrize("d", [0.5, 0.35])
@pytest.mark.parametrize("state", ["plain", "edges", "ungauged"])
def test_fused_step_tracks_the_strict_one(sides, bc, d, state):
    from axions_gb300 import lattice
    from axions_gb300.params import F64_FAST
    rng = np.random.default_rng(6)
    ic = np.array(lattice.random_phase_ic(_params(sides, bc, d, 0), 5))
    if state != "ungauged":
        ic[2:] = rng.uniform(-4, 4, ic[2:].shape)
    if state == "edges":
        pick = rng.random(ic.shape[1:])
        ic[:2, pick < 0.05] = 0.0
        ic[:2, (pick > 0.2) & (pick < 0.3)] *= 1e-30
        ic[2:, pick > 0.8] = 0.0
    want, wdiag = _run(lattice, _params(sides, bc, d, 0, 1), ic)
    got, gdiag = _run(lattice, _params(sides, bc, d, F64_FAST), ic)
    # nine steps of some tens of roundings each
    for c in range(5):
        assert np.linalg.norm(got[c] - want[c]) <= 2e-14 * np.linalg.norm(want[c])
    np.testing.assert_allclose(gdiag, wdiag, rtol=1e-11)


@pytest.mark.parametrize("value", [np.inf, np.nan, 1e200])
@pytest.mark.parametrize("component", [0, 3])
def test_values_out_of_range(value, component):
    from axions_gb300 import lattice
    from axions_gb300.params import F64_FAST
    sides = (34, 32, 36)
    ic = np.array(lattice.random_phase_ic(_params(sides, 0, 0.5, 0), 5))
    ic[2:] = 0.3
    if component < 2 or not np.isfinite(value):
        ic[component].reshape(sides)[7, 9, 11] = value
    want, _ = _run(lattice, _params(sides, 0, 0.5, 0, 1), ic, steps=3)
    got, _ = _run(lattice, _params(sides, 0, 0.5, F64_FAST), ic, steps=3)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))


@pytest.mark.parametrize("sides,bc", [((31, 32, 33), 0), ((32, 32, 32), 0), ((41, 37, 33), 1)])
def test_fields_do_not_depend_on_the_diagnostics(sides, bc):
    from axions_gb300 import lattice
    from axions_gb300.params import F64_FAST
    p = _params(sides, bc, 0.5, F64_FAST)
    ic = np.array(lattice.random_phase_ic(p, 5))
    res = []
    for every in (0, 1, 3):
        with lattice.Lattice(p) as lat:
            lat.set_state(ic, ic, 0)
            lat.advance(7, diag_every=every)
            res.append(lat.get_slots())
    assert np.array_equal(res[0], res[1]) and np.array_equal(res[0], res[2])
