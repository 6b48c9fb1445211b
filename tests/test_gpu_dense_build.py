"""Scene builds from dense device grids against the oracle's build.

The build kernels take 32 bricks per block with wide loads where the grid's
base allows them; sizes here leave partial blocks, put block borders inside
rows of bricks and start the grid off every alignment.
"""
import ctypes

import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


def build(ctx, kind, g, offset):
    """Scene of the grid g, copied to a device address `offset` elements past an aligned one."""
    nz, ny, nx = g.shape
    flat = np.zeros(offset + g.size, dtype=g.dtype)
    flat[offset:] = g.reshape(-1)
    d = ctx.to_device(flat)
    h = ctypes.c_void_p()
    meso._check(meso._lib.meso_scene_create_grid(ctx.handle, kind, d.ptr + offset * g.itemsize, nx, ny, nz, 3,
                                                 ctypes.byref(h)))
    return meso.Scene(ctx, h.value)


@pytest.mark.parametrize("dims", [(32, 32, 32), (96, 32, 64), (160, 96, 32), (352, 64, 96)])
@pytest.mark.parametrize("dtype,kind", [(np.uint8, meso.SRC_GRID_U8), (np.uint16, meso.SRC_GRID_U16)])
@pytest.mark.parametrize("offset", [0, 1, 4, 7])
def test_build_matches_oracle(ctx, dims, dtype, kind, offset):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + offset)
    top = np.iinfo(dtype).max
    # single voxels at any place of a brick, empty bricks, and a solid corner
    g = ((rng.random((nz, ny, nx)) < 0.002) * rng.integers(1, top + 1, (nz, ny, nx))).astype(dtype)
    g[:9, :17, :10] = rng.integers(1, top + 1, (9, 17, 10))
    scene = build(ctx, kind, g, offset)
    bm = oracle.HostBrickMap.from_dense(g.astype(np.uint16))
    ptr, occ, mat = scene.download()
    n = int(scene.info().n_bricks)
    assert np.array_equal(ptr, bm.ptr())
    assert np.array_equal(occ[:n], bm.occ())
    assert np.array_equal(mat[:n], bm.mat())
    scene.destroy()


def test_empty_grid(ctx):
    scene = build(ctx, meso.SRC_GRID_U16, np.zeros((32, 64, 32), np.uint16), 0)
    assert int(scene.info().n_bricks) == 0
    assert (scene.download()[0] == meso.EMPTY_BRICK).all()
    scene.destroy()


@pytest.mark.parametrize("dims", [(32, 32, 32), (96, 64, 32), (512, 512, 64), (512, 512, 544)])
def test_bricks_are_numbered_in_order(ctx, dims):
    # words of 32 bricks: fewer than a thread of the scan takes, fewer than one
    # tile (8192), and more than one with a rest
    nx, ny, nz = dims
    rng = np.random.default_rng(nz)
    keep = rng.random((nz // 8, ny // 8, nx // 8)) < 0.4
    g = np.zeros(dims[::-1], dtype=np.uint8)
    z, y, x = np.nonzero(keep)
    g[8 * z + rng.integers(0, 8, z.size), 8 * y + rng.integers(0, 8, z.size), 8 * x + rng.integers(0, 8, z.size)] = 1
    scene = build(ctx, meso.SRC_GRID_U8, g, 0)
    k = keep.reshape(-1)
    assert np.array_equal(scene.download()[0], np.where(k, np.cumsum(k) - 1, meso.EMPTY_BRICK).astype(np.uint32))
    assert int(scene.info().n_bricks) == k.sum()
    scene.destroy()
