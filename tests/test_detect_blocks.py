"""Crossings of noise and of a smoother level against the oracle, bit for bit, on
lattices of few and of many detection blocks (one or four sites a thread, the change
at 311,296 sites), of less than a block and of blocks that end inside a row; a list
shorter than the crossings gets the first of them."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides,bc", [((3, 3, 3), 0), ((7, 9, 5), 1), ((16, 16, 16), 0), ((33, 17, 29), 0), ((68, 68, 67), 0),
                                      ((68, 68, 68), 0), ((69, 70, 71), 1)])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("steps", [0, 12])
def test_crossings_are_the_oracle_s(oracle_mod, sides, bc, precision, steps):
    from axions_gb300 import lattice
    from axions_gb300.params import LAT_ERR_CAPACITY, make_params
    nx, ny, nz = sides
    p = make_params(0, nx=nx, ny=ny, nz=nz, d=0.5, dt=0.1, lam=2.0, g=0.8, alpha=3.0, bc=bc, precision=precision)
    with lattice.Lattice(p) as lat:
        lat.random_phase_ic_device(4)
        lat.advance(steps)
        st = np.array(lat.get_slots(), dtype=np.float64)
        want = oracle_mod.detect(p, st, steps, 0)
        assert lat.count_crossings() == len(want)
        assert np.array_equal(lat.detect(), want)
        n = len(want) * 2 // 3
        if n:
            buf = np.zeros((n, 3))
            count = ctypes.c_int64(0)
            rc = lat.L.lat_detect_crossings(lat.h, 0, buf.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), n, ctypes.byref(count))
            assert rc == LAT_ERR_CAPACITY and count.value == len(want) and np.array_equal(buf, want[:n])


def test_small_levels_are_spread_over_the_gpu():
    """Counting a noise level of 16^3 takes less than half the time of 64^3, which
    has 64 times the faces (0.36 of it; with the blocks of large lattices 0.68)."""
    from axions_gb300 import lattice
    from axions_gb300.params import make_params
    us = {}
    for n in (16, 64):
        p = make_params(0, nx=n, ny=n, nz=n, d=0.5, dt=0.1, lam=2.0, g=1.0)
        with lattice.Lattice(p) as lat:
            lat.random_phase_ic_device(3)
            lat.count_crossings()
            runs = []
            for _ in range(30):
                t = time.perf_counter()
                lat.count_crossings()
                runs.append(time.perf_counter() - t)
            us[n] = min(runs)
    assert us[16] < 0.5 * us[64], us
