"""Chunks of dense grids against the oracle where their faces depend on the
voxels beside them: on the grid's border, between chunks, with content in the
neighbours' nearest columns only, one and many chunks to a launch, and values
whose only set bit is the lowest or the highest."""
import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,kind,ref_kind,values", [
    (np.uint8, meso.SRC_GRID_U8, oracle.SRC_GRID_U8, [1, 128, 255]),
    (np.uint16, meso.SRC_GRID_U16, oracle.SRC_GRID_U16, [1, 128, 256, 32768])])
@pytest.mark.parametrize("dims", [(32, 32, 32), (64, 32, 32), (32, 64, 96), (96, 32, 64), (160, 64, 32)])
@pytest.mark.parametrize("fill", [0.02, 0.5, 1.0])
def test_neighbours(ctx, dims, dtype, kind, ref_kind, values, fill):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + 2 * ny + 3 * nz)
    g = (rng.choice(np.array(values), (nz, ny, nx)) * (rng.random((nz, ny, nx)) < fill)).astype(dtype)
    # planes beside chunk borders full, empty, and full in every other row
    for x, v in ((31, values[0]), (32, 0), (63, values[-1]), (95, 0), (127, values[0])):
        if x < nx:
            g[:, ::2, x] = v
    coords = np.array([(x, y, z) for z in range(nz // 32) for y in range(ny // 32) for x in range(nx // 32)], dtype=np.int32)
    d = ctx.to_device(g)
    for pick in (slice(None), slice(0, 1), slice(-1, None)):
        q, _ = ctx.mesh(kind, d, coords=coords[pick], dims=dims)
        assert np.array_equal(np.sort(q), oracle.mesh_chunks(ref_kind, g, coords=coords[pick]))
