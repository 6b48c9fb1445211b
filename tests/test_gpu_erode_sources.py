"""The erosion pyramid of every source kind against the oracle: chunk arrays,
grids that start on 16 bytes (wide loads) and that do not (voxel by voxel),
brick maps with and without empty bricks; every depth, content on the chunks'
borders, and values whose only set bit is the lowest or the highest.
"""
import ctypes

import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu

DIMS = (96, 64, 64)


def content(seed, values):
    """Mostly solid, so that some of it lasts several steps: holes, an empty slab, single voxels."""
    rng = np.random.default_rng(seed)
    g = rng.choice(np.array(values), DIMS[::-1])
    holes = rng.integers(0, 32 * 64 * 96, 60)
    g.reshape(-1)[holes] = 0
    g[32:48, 8:24, :] = 0
    g[40, 10, ::7] = values[0]
    g[:, :, 64:72] = 0
    return g


def erode(ctx, kind, data, offset, coords, depth, scene=None):
    """Pyramids of the chunks at coords, the data `offset` elements past an aligned address."""
    src = meso.MeshSource()
    src.kind = kind
    keep = None
    if scene is not None:
        src.scene = scene.handle
    else:
        flat = np.zeros(offset + data.size, dtype=data.dtype)
        flat[offset:] = data.reshape(-1)
        keep = ctx.to_device(flat)
        src.d_data = keep.ptr + offset * data.itemsize
        src.nx, src.ny, src.nz = DIMS
    c = ctx.to_device(np.ascontiguousarray(coords, dtype=np.int32))
    out = ctx.alloc(len(coords) * depth * 4096)
    meso._check(meso._lib.meso_erode_mips(ctx.handle, ctypes.byref(src), c.ptr, len(coords), depth, out.ptr, None))
    ctx.sync()
    w = out.download(np.uint32, len(coords) * depth * 1024).reshape(len(coords), depth, 32, 32)
    return ((w[..., None] >> np.arange(32, dtype=np.uint32)) & 1).astype(np.uint8)


@pytest.mark.parametrize("depth", [1, 2, 5, 8])
@pytest.mark.parametrize("kind,dtype,offset", [(meso.SRC_GRID_U8, np.uint8, 0), (meso.SRC_GRID_U8, np.uint8, 1),
                                               (meso.SRC_GRID_U8, np.uint8, 8), (meso.SRC_GRID_U16, np.uint16, 0),
                                               (meso.SRC_GRID_U16, np.uint16, 1), (meso.SRC_GRID_U16, np.uint16, 8),
                                               (meso.SRC_BRICKMAP, np.uint16, 0)])
def test_grids_and_brick_maps(ctx, kind, dtype, offset, depth):
    g = content(depth, [1, 128, 255] if dtype == np.uint8 else [1, 256, 32768, 65535]).astype(dtype)
    coords = [(x, y, z) for z in (1, 0) for y in range(2) for x in (2, 0, 1)]
    scene = ctx.scene_from_dense(g) if kind == meso.SRC_BRICKMAP else None
    got = erode(ctx, kind, g, offset, coords, depth, scene)
    for i, (x, y, z) in enumerate(coords):
        chunk = g[32 * z:32 * z + 32, 32 * y:32 * y + 32, 32 * x:32 * x + 32]
        assert np.array_equal(got[i], oracle.erode_mips(np.ascontiguousarray(chunk), depth)), (x, y, z)
    if depth < 5:
        assert got[:, -1].any()
    if scene is not None:
        scene.destroy()


@pytest.mark.parametrize("depth", [1, 2, 5, 8])
@pytest.mark.parametrize("kind,dtype", [(meso.SRC_CHUNKS_U8, np.uint8), (meso.SRC_CHUNKS_U16, np.uint16)])
def test_chunk_arrays(ctx, kind, dtype, depth):
    g = content(17 + depth, [1, 128, 255] if dtype == np.uint8 else [1, 256, 32768, 65535]).astype(dtype)
    chunks = g.reshape(2, 32, 2, 32, 3, 32).transpose(0, 2, 4, 1, 3, 5).reshape(-1, 32, 32, 32)
    got = ctx.erode_mips(kind, ctx.to_device(np.ascontiguousarray(chunks)), n=len(chunks), depth=depth)
    bits = ((got[..., None] >> np.arange(32, dtype=np.uint32)) & 1).astype(np.uint8)
    for i, chunk in enumerate(chunks):
        assert np.array_equal(bits[i], oracle.erode_mips(chunk, depth)), i


def test_chunks_outside_are_flagged_and_empty(ctx):
    g = np.full(DIMS[::-1], 3, dtype=np.uint8)
    with pytest.raises(meso.MesoError):
        erode(ctx, meso.SRC_GRID_U8, g, 0, [(0, 0, 0), (3, 0, 0)], 2)
    got = erode(ctx, meso.SRC_GRID_U8, g, 0, [(0, 0, 0)], 2)  # the flag is cleared
    assert got[0, 0].all() and got[0, 1].sum() == 30 ** 3
