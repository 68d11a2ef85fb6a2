"""The random-phase initial state of an FP32 lattice, whose sines and cosines
come from the integer pipe, is the FP64 lattice's (CUDA's) rounded to floats,
value for value; amplitudes include tiny ones, whose floats are subnormal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("eta", [1.0, 0.7, 1e-37, 3e38])
@pytest.mark.parametrize("n", [3, 160])
def test_fp32_state_is_the_fp64_one_rounded(model, eta, n):
    from axions_gb300 import lattice
    from axions_gb300.params import F32, make_params
    got = []
    for precision in (0, F32):
        p = make_params(model, n=n, d=0.5, dt=0.1, lam=2.0, g=1.0, eta=eta, damped_nt=0, alpha=3.0, precision=precision,
                        **({"lambda2": 2.0, "q1": 1.0, "q2": 2.0, "eta2": 0.9} if model else {}))
        with lattice.Lattice(p) as lat:
            lat.random_phase_ic_device(12345, independent=True)
            got.append(lat.get_slots())
    with np.errstate(over="ignore"):
        want = got[0].astype(np.float32).astype(np.float64)
    assert np.array_equal(got[1], want)
