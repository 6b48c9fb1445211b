"""Rays that meet a brick whose pointer an edit has taken away before its level byte.

An edit unlinks bricks first and rebuilds the maps derived from the pointers in a
later launch, so a view on a stream that is not ordered with the edit can see an
occupied level and no slot.  It must then read no slot (the pointer's value lies
tens of gigabytes past the pools).  The state is made here by taking pointers out
of the grid by hand, on the views' own stream.
"""
import ctypes

import numpy as np
import pytest

import mesoengine_gb300 as meso

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shadow", [False, True])
@pytest.mark.parametrize("views", [1, 3, 40])
def test_unlinked_bricks_are_empty(ctx, views, shadow):
    t = meso.terrain_preset("small")
    scene = ctx.scene_from_terrain(t)
    nx, ny, _ = scene.dims
    poses = [(-60.0, -50.0, 150.0), (200.0, 160.0, 120.0), (64.0, 64.0, 90.0)]
    cams = [meso.camera(poses[k % 3], (64.0, 64.0, 20.0), 120, 80) for k in range(views)]
    full = ctx.raymarch(scene, cams, shadow=shadow)

    def brick(h):
        v = h["voxel"].astype(np.int64)
        return v % nx // 8 + (nx // 8) * (v // nx % ny // 8 + (ny // 8) * (v // (nx * ny) // 8))

    hit = np.isfinite(full["t"])
    seen = np.unique(brick(full[hit]))
    gone = seen[::3]
    assert gone.size > 30
    ptr, _, _ = scene.download()
    cut = ptr.copy()
    cut[gone] = meso.EMPTY_BRICK
    d_ptr = scene.info().d_ptr

    def put(p):
        meso._check(meso.load().meso_memcpy_h2d(ctx.handle, ctypes.c_void_p(d_ptr), meso._np_ptr(p), p.nbytes, None))
        ctx.sync()

    put(cut)
    got = ctx.raymarch(scene, cams, shadow=shadow)
    put(ptr)
    in_gone = np.zeros(full.size, bool)
    in_gone[hit] = np.isin(brick(full[hit]), gone)
    again = np.isfinite(got["t"])
    assert not np.isin(brick(got[again]), gone).any()
    assert (got["t"][in_gone] >= full["t"][in_gone]).all()
    if not shadow:  # a ray that hit another brick takes the same way, past or through the ones that are gone
        assert np.array_equal(got[~in_gone].view(np.uint8), full[~in_gone].view(np.uint8))
    assert np.array_equal(ctx.raymarch(scene, cams, shadow=shadow).view(np.uint8), full.view(np.uint8))
    scene.destroy()
