"""Views into host memory with every shape of block.

Views into page-locked memory take their own blocks (tiles in a row, whole rows
written at once where four warps of 8x4 tiles allow it) in an order of their own.
"""
import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu

POSE = ((-31.0, -17.0, 90.0), (48.0, 80.0, 32.0))
# one tile and less, ends inside a tile and a row of tiles, rows that start on 16 bytes and that do
# not, and sizes with enough blocks that their order strides over them
SIZES = [(1, 1), (7, 3), (33, 9), (64, 32), (65, 33), (3, 70), (32, 4), (320, 200), (8, 2050)]


@pytest.mark.parametrize("tile_w", [4, 8, 16, 32])
@pytest.mark.parametrize("warps", [1, 2, 3, 4])
def test_every_block_shape_into_host_memory(warps, tile_w):
    rng = np.random.default_rng(8)
    g = np.zeros((64, 160, 96), np.uint16)
    for _ in range(40):
        x, y, z = (int(rng.integers(0, n)) for n in (96, 160, 64))
        g[z:z + 9, y:y + 14, x:x + 11] = rng.integers(1, 65536)
    bm = oracle.HostBrickMap.from_dense(g)
    c = meso.Context(0, ray_warps_per_cta=warps, ray_tile_w=tile_w, ray_tile_h=32 // tile_w)
    scene = c.scene_from_dense(g)
    pinned = c.pinned(24 * max(w * h for w, h in SIZES) + 8)
    for w, h in SIZES:
        ref = oracle.raymarch(bm, oracle.camera(*POSE, w, h)).view(np.uint8)
        for offset in (0, 8):
            c.raymarch_host(scene, meso.camera(*POSE, w, h), out_ptr=pinned.ptr + offset)
            got = pinned.view(np.uint8, 24 * w * h + offset)[offset:]
            assert np.array_equal(got, ref), (w, h, offset)
        assert np.array_equal(c.raymarch_host(scene, meso.camera(*POSE, w, h)).view(np.uint8), ref)
    scene.destroy()
    c.close()
