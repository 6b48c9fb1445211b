"""Brick-map lists of every ticket size.

A CTA takes up to 8 list entries to a ticket, as many as leave it 8 tickets, and
tests them together against the scene's cell map: entries with invalid coordinates,
air chunks that are counted without being meshed, and the permutation of the list
(whose multiplier is another one for lists of a multiple of 7919) are looked at
with tickets of every size.  The lengths follow from the device's SMs.
"""
import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup():
    c = meso.Context(0, mesh_ctas_per_sm=1)
    scene = c.scene_from_terrain(meso.terrain_preset("small"))
    chunks = np.array([(x, y, z) for z in range(4) for y in range(4) for x in range(4)], dtype=np.int32)
    ref = oracle.mesh_chunks(oracle.SRC_BRICKMAP, coords=chunks, bm=oracle.HostBrickMap.from_dense(scene.dense()))
    which = (ref >> np.uint64(44)).astype(np.int64)
    yield c, scene, chunks, [ref[which == k] & np.uint64((1 << 44) - 1) for k in range(64)]
    scene.destroy()
    c.close()


@pytest.mark.parametrize("size", [1, 2, 3, 5, 7, 8, 9, "7919", "2 x 7919"])
def test_tickets(setup, size):
    c, scene, chunks, quads = setup
    n = {"7919": 7919, "2 x 7919": 15838}.get(size) or 8 * c.sm_count * size + 5
    rng = np.random.default_rng(n)
    pick = rng.integers(0, 64, n)
    coords = chunks[pick]
    bad = rng.choice(n, 4, replace=False)
    coords[bad] = [(4, 0, 0), (0, -1, 0), (0, 0, 4), (-1, 9, 2)]
    lists = [quads[k] for k in pick]
    for b in bad:
        lists[b] = quads[0][:0]
    counts_ref = np.array([q.size for q in lists])
    ref = np.concatenate(lists) | (np.repeat(np.arange(n, dtype=np.uint64), counts_ref) << np.uint64(44))
    with pytest.raises(meso.MesoError, match="outside"):
        c.mesh(meso.SRC_BRICKMAP, coords=coords, scene=scene, capacity=ref.size)
    got, counts = c.mesh(meso.SRC_BRICKMAP, coords=coords, scene=scene, capacity=ref.size, chunk_counts=True, check=False)
    assert np.array_equal(counts, counts_ref)
    assert (counts_ref[np.setdiff1d(np.arange(n), bad)] == 0).sum() > n // 20  # air chunks among them
    assert np.array_equal(np.sort(got), np.sort(ref))
