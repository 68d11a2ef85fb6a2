"""A level at rest has no Gauss deviation: with both levels the same, every kernel's
first diagnostic is exactly 0, also where the spacings round (the past level's
divergence comes from another kernel than the step's)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("sides,bc", [((12, 10, 64), 0), ((12, 18, 32), 0), ((9, 11, 33), 0), ((9, 10, 66), 1), ((16, 12, 36), 0)])
@pytest.mark.parametrize("d", [(0.5, 0.5, 0.5), (0.35, 0.35, 0.35), (0.5, 0.4, 0.35)])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_static_levels(model, sides, bc, d, precision):
    from axions_gb300 import lattice
    from axions_gb300.params import F32, make_params
    kw = dict(lambda2=2.0, lambda12=0.0, eta2=1.0, q1=1.0, q2=2.0) if model else {}
    rng = np.random.default_rng(3)
    for variant in (0, 2, 3) if precision == F32 else (0,):
        p = make_params(model, nx=sides[0], ny=sides[1], nz=sides[2], dx=d[0], dy=d[1], dz=d[2], dt=0.05, lam=2.0, g=0.7, bc=bc,
                        precision=precision, kernel_variant=variant, **kw)
        with lattice.Lattice(p) as lat:
            ic = np.array(lattice.random_phase_ic(p, 3))
            ic[-3:] = rng.uniform(-1, 1, ic[-3:].shape)
            lat.set_state(ic, ic, 0)
            assert lat.diagnostics().gauss_abs_sum == 0.0, variant
            assert lat.advance(1, diag_every=1)[0][2] == 0.0, variant
            if precision == F32 and variant == 0:
                lat.set_state(ic, ic, 0)
                with lattice.Batch(1) as b:
                    b.add(lat, diag_every=1, stop_step=1)
                    b.advance(1)
                    assert b.take_diags(lat)[0][2] == 0.0
