"""The raymarch's region walk against the oracle's step-by-step walk.

The kernel leaves aligned empty cubes of 1 to 512 voxels on a side in one
step each and counts the steps it passed over from the positions; every field
of every hit, t included, has to be the same bytes as the oracle's, for every
direction octant, for directions with zero components, for origins on voxel,
brick and chunk boundaries (boundary times that tie), for grids whose sides
are no multiple of a cell, after edits and after a load, and for the values
that take the step-by-step path instead (far cameras, a light without a
direction).
"""
import ctypes

import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


def same(got, ref):
    bad = np.nonzero((got.view(np.uint8).reshape(-1, 24) != ref.view(np.uint8).reshape(-1, 24)).any(1))[0]
    assert bad.size == 0, f"{bad.size} of {got.size} hits differ, first {got[bad[:3]]} vs {ref[bad[:3]]}"


def sparse(dims, seed, n_points, n_boxes):
    """A mostly empty grid: single voxels, and boxes of a few voxels to a few bricks."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    g = np.zeros((nz, ny, nx), dtype=np.uint16)
    for _ in range(n_points):
        g[rng.integers(nz), rng.integers(ny), rng.integers(nx)] = rng.integers(1, 65536)
    for _ in range(n_boxes):
        x, y, z = (int(rng.integers(0, n)) for n in dims)
        w, h, d = (int(v) for v in rng.integers(1, 20, 3))
        g[z:z + d, y:y + h, x:x + w] = rng.integers(1, 65536)
    return g


@pytest.fixture(scope="module", params=[((32, 32, 32), 60, 2), ((96, 160, 64), 60, 12), ((544, 288, 320), 80, 60),
                                        ((1024, 64, 576), 60, 40)], ids=lambda p: "x".join(map(str, p[0])))
def grid(ctx, request):
    dims, points, boxes = request.param
    g = sparse(dims, sum(dims), points, boxes)
    scene = ctx.scene_from_dense(g)
    yield dims, scene, oracle.HostBrickMap.from_dense(g)
    scene.destroy()


def both(ctx, scene, bm, o, target, w=56, h=37, light=None):
    same(ctx.raymarch(scene, meso.camera(o, target, w, h), light=light),
         oracle.raymarch(bm, oracle.camera(o, target, w, h), light=light))


def test_every_octant(ctx, grid):
    dims, scene, bm = grid
    c = [n / 2.0 + 0.37 for n in dims]
    for k in range(8):
        s = [1 if (k >> a) & 1 else -1 for a in range(3)]
        out = [c[a] - s[a] * (0.6 * dims[a] + 21.3) for a in range(3)]
        into = [c[a] + s[a] * (0.4 * dims[a] + 5.1) for a in range(3)]
        both(ctx, scene, bm, out, c)   # from outside
        both(ctx, scene, bm, c, into)  # from inside
        light = np.array([0.3 * s[0], 0.5 * s[1], 0.8 * s[2]], dtype=np.float32)
        both(ctx, scene, bm, out, c, light=light)


def test_ties_and_axis_aligned_rays(ctx, grid):
    dims, scene, bm = grid
    nx, ny, nz = dims
    # an odd image size puts rays exactly along the axis through its middle
    for o, target in [((nx / 2, ny / 2, nz + 40.0), (nx / 2, ny / 2, 0.0)), ((-33.0, ny / 2, nz / 2), (nx, ny / 2, nz / 2)),
                      ((nx / 2, ny + 8.0, nz / 2), (nx / 2, 0.0, nz / 2)), ((0.0, 0.0, 0.0), (nx, ny, nz)),
                      ((float(nx), float(ny), float(nz)), (0.0, 0.0, 0.0)), ((-32.0, -32.0, -32.0), (32.0, 32.0, 32.0)),
                      ((nx - 0.5, 0.5, 0.5), (nx - 33.5, 33.5, 33.5)), ((nx / 2, ny / 2, nz / 2), (nx / 2 + 8, ny / 2 + 8, nz / 2))]:
        for w, h in ((33, 33), (32, 32)):
            both(ctx, scene, bm, o, target, w, h)
    for light in ((0.0, 0.0, 1.0), (1.0, 0.0, 0.0), (0.0, -1.0, 0.0), (1.0, 1.0, 1.0), (-0.5, 0.0, 0.5), (1e3, 2e3, 1e3)):
        both(ctx, scene, bm, (-31.0, -17.0, nz + 25.0), (nx / 2, ny / 2, nz / 2), light=np.array(light, np.float32))


def test_values_off_the_region_path(ctx, grid):
    dims, scene, bm = grid
    nx, ny, nz = dims
    mid = (nx / 2, ny / 2, nz / 2)
    both(ctx, scene, bm, (-140000.0, ny / 2 + 3.0, nz / 2 + 1.0), mid, 16, 9)  # beyond the region path's coordinates
    both(ctx, scene, bm, (-100000.0, ny / 2 + 3.0, nz / 2 + 1.0), mid, 16, 9)  # within them
    for light in ((0.0, 0.0, 0.0), (1e-32, 0.0, 1.0), (0.0, 1e-36, 0.0), (1e31, 1e31, 1e31)):
        both(ctx, scene, bm, (-31.0, -17.0, nz + 25.0), mid, 24, 17, light=np.array(light, np.float32))
    # a view that needs the step-by-step path beside one that does not
    cams = [((-31.0, -17.0, nz + 25.0), mid), ((-140000.0, ny / 2 + 3.0, nz / 2 + 1.0), mid)]
    got = ctx.raymarch(scene, [meso.camera(o, t, 20, 11) for o, t in cams])
    same(got, oracle.raymarch(bm, [oracle.camera(o, t, 20, 11) for o, t in cams]))


def _edits(rng, dims, n, radius):
    return [(tuple(int(rng.integers(0, d)) for d in dims), int(rng.integers(0, radius + 1)),
             0 if rng.random() < 0.4 else int(rng.integers(1, 65536))) for _ in range(n)]


@pytest.mark.parametrize("radius", [0, 1, 3, 40])
def test_maps_follow_edits(ctx, radius, tmp_path):
    # single voxels and small spheres (blocks inside bricks), large ones
    # (cells of every level emptied and filled); then the same scene from a file
    dims = (544, 288, 320)
    g = sparse(dims, 7, 200, 30)
    scene, bm = ctx.scene_from_dense(g, spare_bricks=20000), oracle.HostBrickMap.from_dense(g)
    rng = np.random.default_rng(radius)
    poses = [((-60.0, -80.0, 400.0), (270.0, 140.0, 100.0)), ((600.0, 350.0, -40.0), (200.0, 100.0, 200.0))]
    for _ in range(3):
        e = _edits(rng, dims, 24, radius)
        scene.edit([meso.SphereEdit((ctypes.c_int32 * 3)(*c), r, m, 0) for c, r, m in e])
        bm.edit([oracle.Sphere((ctypes.c_int32 * 3)(*c), r, m, 0) for c, r, m in e])
        for o, t in poses:
            both(ctx, scene, bm, o, t, 120, 80)
    path = str(tmp_path / "scene.bin")
    scene.save(path)
    again = ctx.scene_load(path)
    for o, t in poses:
        both(ctx, again, bm, o, t, 120, 80)
    again.destroy()
    scene.destroy()


@pytest.mark.parametrize("tile_w", [4, 8, 16, 32])
@pytest.mark.parametrize("warps", [1, 2, 3, 4])
def test_every_block_shape(ctx, warps, tile_w):
    # images that end inside a tile, a row of tiles and a block, of one tile
    # and of less; one view, several as parameters, and a table of them
    g = sparse((96, 160, 64), 5, 60, 12)
    bm = oracle.HostBrickMap.from_dense(g)
    c = meso.Context(0, ray_warps_per_cta=warps, ray_tile_w=tile_w, ray_tile_h=32 // tile_w)
    scene = c.scene_from_dense(g)
    pose = ((-31.0, -17.0, 90.0), (48.0, 80.0, 32.0))
    sizes = [(1, 1), (7, 3), (33, 9), (64, 32), (65, 33), (3, 70)]
    for n in (1, len(sizes), 36):
        cams = [sizes[k % len(sizes)] for k in range(n)]
        got = c.raymarch(scene, [meso.camera(*pose, w, h) for w, h in cams])
        same(got, oracle.raymarch(bm, [oracle.camera(*pose, w, h) for w, h in cams]))
    scene.destroy()
    c.close()


@pytest.mark.parametrize("lo,hi", [((0, 0, 0), (32, 32, 32)), ((64, 96, 32), (96, 160, 64)), ((130, 70, 40), (131, 71, 41)),
                                   ((0, 128, 0), (256, 160, 96)), ((200, 0, 90), (256, 192, 96)), (None, None)])
def test_space_outside_the_bounds(ctx, lo, hi):
    # content in one part of the grid (a corner cell, an inner box, one voxel,
    # slabs along faces, none): rays that enter its bounds from each side and
    # from inside, that miss them, that pass along their faces and corners;
    # then bounds that edits widen, and that keep their size as edits empty them
    dims = (256, 192, 96)
    rng = np.random.default_rng(11)
    g = np.zeros(dims[::-1], dtype=np.uint16)
    if lo is not None:
        part = g[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]]
        part[...] = (rng.random(part.shape) < 0.02) * 9
        part.flat[0] = part.flat[-1] = 3
    lo, hi = lo or (96, 96, 32), hi or (128, 128, 64)
    scene, bm = ctx.scene_from_dense(g, spare_bricks=2000), oracle.HostBrickMap.from_dense(g)
    mid = [(a + b) / 2.0 for a, b in zip(lo, hi)]
    face = [32.0 * (a // 32) for a in lo]  # of the cell that the lowest voxel is in

    def look():
        for k in range(8):
            s = [1 if (k >> a) & 1 else -1 for a in range(3)]
            both(ctx, scene, bm, [mid[a] - s[a] * (0.7 * dims[a] + 9.3) for a in range(3)], mid, 40, 30)
            both(ctx, scene, bm, [dims[a] * (0.5 - 0.45 * s[a]) for a in range(3)], mid, 40, 30,
                 light=np.array([0.3 * s[0], 0.5 * s[1], 0.8 * s[2]], np.float32))
        both(ctx, scene, bm, mid, [0.0, 0.0, 0.0], 40, 30)
        for a in range(3):  # in the plane of a face of the bounds, and through its corner
            d = [40.0 * (b != a) for b in range(3)]
            both(ctx, scene, bm, [f - v for f, v in zip(face, d)], face, 33, 33)
        both(ctx, scene, bm, [f - 40.0 for f in face], face, 33, 33)

    look()
    scene.edit([meso.SphereEdit((ctypes.c_int32 * 3)(20, 30, 80), 5, 7, 0)])
    bm.edit([oracle.Sphere((ctypes.c_int32 * 3)(20, 30, 80), 5, 7, 0)])
    look()
    whole = [((x, y, z), 70, 0) for x in (0, 85, 170, 255) for y in (0, 95, 191) for z in (0, 95)]
    scene.edit([meso.SphereEdit((ctypes.c_int32 * 3)(*c), r, m, 0) for c, r, m in whole])
    bm.edit([oracle.Sphere((ctypes.c_int32 * 3)(*c), r, m, 0) for c, r, m in whole])
    look()
    scene.destroy()
