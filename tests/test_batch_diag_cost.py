"""Batched steps with diagnostics at every step cost less than 1.85 plain ones where
the batch fills the GPU (64 lattices of 32^3: 1.69; with FP64 conversions and two full
trees of additions for every partial sum 2.02), and their sums agree with a single
lattice's."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_diagnostics_at_every_step():
    from axions_gb300 import lattice
    from axions_gb300.params import F32, make_params
    p = make_params(0, nx=32, ny=32, nz=32, d=0.5, dt=0.1, lam=2.0, g=1.0, alpha=3.0, precision=F32)
    us, sums = {}, {}
    for every in (0, 1):
        lats = [lattice.Lattice(p) for _ in range(64)]
        with lattice.Batch(64) as b:
            for s, lat in enumerate(lats):
                lat.random_phase_ic_device(s)
                b.add(lat, diag_every=every, stop_step=10 ** 6)
            runs = []
            for _ in range(12):
                t = time.perf_counter()
                b.advance(50)
                runs.append(time.perf_counter() - t)
            us[every] = min(runs) / 50 * 1e6
            sums[every] = b.take_diags(lats[5])
        for lat in lats:
            lat.close()
    assert us[1] < 1.85 * us[0], us
    with lattice.Lattice(p) as lat:
        lat.random_phase_ic_device(5)
        want = np.array(lat.advance(20, diag_every=1))
    np.testing.assert_allclose(np.array(sums[1])[:20], want, rtol=1e-6)
