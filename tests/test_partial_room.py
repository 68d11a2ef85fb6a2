"""The room of a lattice's diagnostic partials (16 bytes each, part of its footprint)
holds one for every CTA of every FP32 tile shape (64x4, 32x8) at one plane a CTA,
whatever shape the lattice is routed to: ragged sides, fixed walls."""
import pytest


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("sides", [(74, 33, 32), (32, 33, 36), (7, 5, 9), (20, 130, 3), (64, 64, 64), (33, 97, 68), (201, 199, 203), (16, 4, 580)])
def test_every_tile_shape_has_room(model, bc, sides):
    from axions_gb300 import lattice
    from axions_gb300.params import F32, make_params
    nx, ny, nz = sides
    p = make_params(model, nx=nx, ny=ny, nz=nz, precision=F32, bc=bc)
    fields = 4 * (2 * (7 if model else 5) + 1) * nx * ny * nz
    room = (lattice.footprint_bytes(p) - fields - 16) // 16   # two counters besides
    x, y, z = (n - 2 * bc for n in sides)
    for tz, ty in ((64, 4), (32, 8)):
        assert room >= x * -(-y // ty) * -(-z // tz), (tz, ty)
