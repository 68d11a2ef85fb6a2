"""The ordered sums of the string length (string_length.cu ChainSum), which add
tiles of 512 values as integers where no addition in the tile rounds to even
on a tie or leaves the sum's binade: bit for bit the oracle's sequential sums
at the edges of the tiles, for lengths that are dyadic (every sum exact), that
repeat one inexact value, and that are random."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 31, 32, 33, 255, 256, 257, 512, 511, 513, 1023, 1500, 4097])
@pytest.mark.parametrize("kind", ["dyadic", "tenths", "random"])
def test_sums_are_the_sequential_ones(oracle_mod, M, kind):
    from axions_gb300 import lattice
    from axions_gb300.params import make_params
    p = make_params(0, nx=40, ny=36, nz=44, d=0.5)
    rng = np.random.default_rng(M)
    lo = -0.5 * np.array([(n - 1) // 2 for n in (40, 36, 44)], dtype=np.float64)
    size = 0.5 * np.array([40, 36, 44])
    if kind == "random":
        pts = lo + rng.random((M, 3)) * size * (0.6 if M > 1000 else 0.25)
    else:
        step = 0.25 if kind == "dyadic" else 0.1
        n = int(np.ceil(M ** (1 / 3))) + 1
        grid = np.stack(np.meshgrid(*(np.arange(n),) * 3, indexing="ij"), -1).reshape(-1, 3)
        pts = (lo + step * grid[rng.permutation(len(grid))[:M]]) + 0.25 * size
    for split in (True, False):
        assert lattice.string_length_points(p, pts, split, lattice.CHAIN_HASH) == oracle_mod.string_length(p, pts, split)
