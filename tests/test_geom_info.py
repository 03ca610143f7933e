"""The device bytes that a geometry reports: all arrays that it keeps."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

TILE, TILE_BYTES = 128, 64  # slots of a tile of the sorted order; its record: 3 integers, 6 doubles


@pytest.mark.parametrize("box, faces, corrections", [
    ((0.5, 0.5, 0.5, 4, 0.2, 4.0, 1.0), [256] * 6, False),   # planes of exactly two tiles
    ((0.5, 0.5, 0.5, 4, 0.2, 4.0, 1.0), [256] * 6, True),
    ((0.7, 0.6, 0.5, 3, 0.3, 4.0, 1.0), None, True),          # small planes: one group, a ragged last tile
])
def test_reported_bytes_cover_every_array(bie, box, faces, corrections):
    from dielectricbie_jl_b200 import _abi
    itf = bie.single_dielectric_box3d(*box)
    if faces:
        assert itf.n == sum(faces)
    near = itf.near(8, 1e-9, True) if corrections else None
    g = bie._Geom(itf, near, 0)
    n, nblocks, got = C.c_int64(), C.c_int64(), C.c_size_t()
    _abi.check(_abi.lib().bie_geom_info(g._h, C.byref(n), C.byref(nblocks), C.byref(got)))
    slots = -(-itf.n // TILE) * TILE
    # positions, normals, weight, diagonal and its reciprocal; sorted positions and weights; node of each slot
    want = 8 * 9 * itf.n + (4 * 8 + 4) * slots + slots // TILE * TILE_BYTES
    if corrections:
        nb = box[3] ** 2
        want += 4 * (itf.npanels + 1 + nblocks.value) + 8 * nblocks.value * nb * nb
    assert n.value == itf.n and got.value == want
