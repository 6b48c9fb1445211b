"""Updates of the resident mesh store whose quads fill part of a warp, one warp or
many: placed, added to and taken away, each segment against the oracle."""
import ctypes

import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


def _coords(dims):
    cx, cy, cz = dims[0] // 32, dims[1] // 32, dims[2] // 32
    idx = np.arange(cx * cy * cz, dtype=np.int64)
    return np.stack([idx % cx, (idx // cx) % cy, idx // (cx * cy)], 1).astype(np.int32)


def _assert_store_matches(store, bm, dims):
    n = (dims[0] // 32) * (dims[1] // 32) * (dims[2] // 32)
    ref = oracle.mesh_chunks(oracle.SRC_BRICKMAP, coords=_coords(dims), bm=bm)
    assert np.array_equal(np.sort(store.gather(np.arange(n))), ref)
    assert store.info().live_quads == len(ref)


@pytest.mark.parametrize("quads", [1, 6, 31, 32, 33, 250])
def test_store_updates_of_few_and_many_quads(ctx, quads):
    """Update lists whose temporary buffer holds one warp's share of quads or a
    remainder, of one chunk and of many chunks with quads side by side: single
    voxels apart from one another, six quads each but on a chunk's border."""
    dims = (128, 96, 64)
    g = np.zeros(dims[::-1], dtype=np.uint16)
    rng = np.random.default_rng(quads)
    cells = rng.permutation(np.stack(np.meshgrid(*[np.arange(1, d, 3) for d in dims[::-1]], indexing="ij"), -1).reshape(-1, 3))
    scene, bm = ctx.scene_from_dense(g, spare_bricks=4000), oracle.HostBrickMap.from_dense(g)
    store = ctx.mesh_store(scene)
    # placed, more of them, then some taken away
    for part, m in ((cells[:(quads + 5) // 6], 7), (cells[:quads], 7), (cells[:(quads + 1) // 2], 0)):
        sp = [([int(c[2]), int(c[1]), int(c[0])], 0, m) for c in part]
        dirty = scene.edit([meso.SphereEdit((ctypes.c_int32 * 3)(*c), r, v, 0) for c, r, v in sp])
        bm.edit([oracle.Sphere((ctypes.c_int32 * 3)(*c), r, v, 0) for c, r, v in sp])
        store.update(dirty)
        _assert_store_matches(store, bm, dims)
    store.destroy()
    scene.destroy()
