"""Views and lights whose values the region walk does not take: results and time.

Cameras more than 2^17 voxels from the grid, and directions with a nonzero
component below 1e-30 or one above 1e30, walk by the definition's own steps.
They cross empty space in cubes all the same; every field of every hit, steps
included, has to be the oracle's, also where the boundary times of neighbouring
bricks round to the same float, and a far view must not pay for each empty brick.
"""
import ctypes

import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


def sparse(dims, seed, boxes):
    rng = np.random.default_rng(seed)
    g = np.zeros(dims[::-1], dtype=np.uint16)
    for _ in range(boxes):
        x, y, z = (int(rng.integers(0, n)) for n in dims)
        w, h, d = (int(v) for v in rng.integers(1, 24, 3))
        g[z:z + d, y:y + h, x:x + w] = rng.integers(1, 65536)
    return g


@pytest.fixture(scope="module", params=[(96, 160, 64), (544, 288, 320), (1024, 64, 576)], ids=lambda p: "x".join(map(str, p)))
def grid(ctx, request):
    dims = request.param
    g = sparse(dims, sum(dims), 30)
    scene = ctx.scene_from_dense(g)
    yield dims, scene, oracle.HostBrickMap.from_dense(g)
    scene.destroy()


def both(ctx, scene, bm, o, target, w, h, tan=None, light=None, shadow=True):
    a, b = meso.camera(o, target, w, h), oracle.camera(o, target, w, h)
    if tan is not None:
        a.tan_half_fov_y = b.tan_half_fov_y = tan
    got = ctx.raymarch(scene, a, light=light, shadow=shadow)
    ref = oracle.raymarch(bm, b, light=light, shadow=shadow)
    bad = np.nonzero((got.view(np.uint8).reshape(-1, 24) != ref.view(np.uint8).reshape(-1, 24)).any(1))[0]
    assert bad.size == 0, f"{bad.size} of {got.size} hits differ, first {got[bad[:3]]} vs {ref[bad[:3]]}"
    return np.isfinite(got["t"]).sum()


@pytest.mark.parametrize("dist", [131100.0, 1e6, 3e7, 2e9])
def test_far_cameras(ctx, grid, dist):
    # from a few thousandths of a voxel between neighbouring floats of a
    # boundary's coordinate (131,100) to hundreds of voxels (2e9)
    dims, scene, bm = grid
    mid = [n / 2.0 + 0.37 for n in dims]
    tan = 0.8 * max(dims) / dist
    hits = 0
    for k in range(8):
        s = [1 if (k >> a) & 1 else -1 for a in range(3)]
        for d in ((1.0, 0.7, 0.4), (0.2, 1.0, 0.05), (0.0, 0.3, 1.0)):
            hits += both(ctx, scene, bm, [mid[a] - s[a] * d[a] * dist for a in range(3)], mid, 48, 33, tan)
    for a in range(3):  # along the axes: components of zero and next to it
        for s in (-1.0, 1.0):
            o = [m - s * dist * (b == a) for b, m in enumerate(mid)]
            hits += both(ctx, scene, bm, o, mid, 33, 33, tan)
    assert hits > 0 or dist > 1e9


@pytest.mark.parametrize("light", [(1e-32, 0.6, 0.8), (0.6, -1e-36, -0.8), (1e-40, 1e-40, 1.0), (0.5, 0.5, -1e-31), (1e31, 1.0, 1e31),
                                   (-1e31, 1e-31, 0.1), (1e-32, 1e-32, 1e-32), (3e38, 0.0, 1e38), (0.0, 0.0, 0.0)])
def test_lights_off_the_region_path(ctx, grid, light):
    dims, scene, bm = grid
    mid = [n / 2.0 for n in dims]
    for o in ((-60.0, -50.0, dims[2] + 70.0), (dims[0] + 40.0, dims[1] + 90.0, -80.0)):
        assert both(ctx, scene, bm, o, mid, 72, 48, light=np.array(light, np.float32)) > 0


def test_edits_and_empty_grids(ctx):
    dims = (544, 288, 320)
    g = sparse(dims, 3, 20)
    scene, bm = ctx.scene_from_dense(g, spare_bricks=100000), oracle.HostBrickMap.from_dense(g)
    o, mid = (-150000.0, 90000.0, 120000.0), (270.0, 140.0, 160.0)
    tan = 400.0 / 210000.0
    rng = np.random.default_rng(5)
    for radius in (2, 30, 200):
        e = [(tuple(int(rng.integers(0, d)) for d in dims), radius, int(rng.integers(0, 3)) * 7) for _ in range(8)]
        scene.edit([meso.SphereEdit((ctypes.c_int32 * 3)(*c), r, m, 0) for c, r, m in e])
        bm.edit([oracle.Sphere((ctypes.c_int32 * 3)(*c), r, m, 0) for c, r, m in e])
        both(ctx, scene, bm, o, mid, 90, 60, tan)
    scene.destroy()
    none = np.zeros((64, 576, 96), np.uint16)
    scene, bm = ctx.scene_from_dense(none), oracle.HostBrickMap.from_dense(none)
    assert both(ctx, scene, bm, (-150000.0, 200.0, 90000.0), (48.0, 288.0, 32.0), 40, 30, 0.003) == 0
    scene.destroy()


@pytest.mark.parametrize("shadow", [False, True])
def test_far_views_beside_near_ones(ctx, grid, shadow):
    # in one launch with its views as parameters, through the tables of more
    # than 32, and through a server's checksum launch; a direction with a tiny
    # component among them
    dims, scene, bm = grid
    mid = [n / 2.0 for n in dims]
    poses = [([-60.0, -50.0, dims[2] + 70.0], None), ([-150000.0, 40000.0, 90000.0], 400.0 / 180000.0),
             ([mid[0] + 0.25, mid[1] + 0.25, dims[2] + 40.0], None)]

    def cams(module, n):
        out = []
        for k in range(n):
            o, tan = poses[k % 3]
            c = module.camera(o, mid, 41, 27)
            if tan is not None:
                c.tan_half_fov_y = tan
            if k % 3 == 2:
                c.forward[0], c.forward[1], c.forward[2], c.tan_half_fov_y = 1e-33, 0.0, -1.0, 0.5 if k % 2 else 0.0
            out.append(c)
        return out

    def same(got, n):
        ref = oracle.raymarch(bm, cams(oracle, n), shadow=shadow)
        assert np.array_equal(got.view(np.uint8).reshape(-1, 24), ref.view(np.uint8).reshape(-1, 24))

    for n in (3, 40):
        same(ctx.raymarch(scene, cams(meso, n), shadow=shadow), n)
        out = ctx.alloc(24 * 41 * 27 * n)
        light = meso._light_arg(None)
        meso._check(meso.load().meso_raymarch_noalloc(ctx.handle, (ctypes.c_void_p * n)(*[scene.handle] * n), (meso.Camera * n)(*cams(meso, n)),
                                                      n, meso._np_ptr(light), int(shadow), out.ptr, None))
        ctx.sync()
        same(out.download(meso.HIT_DTYPE, 41 * 27 * n), n)
    srv = meso.Server(ctx, [scene], max_inflight_batches=1, max_batch_rays=1 << 20)
    bufs = [ctx.alloc(24 * 41 * 27) for _ in range(6)]
    for k, c in enumerate(cams(meso, 6)):
        srv.submit(0, c, shadow=shadow, tag=k, dst=bufs[k])
    srv.drain(20.0)
    assert all(c.status == 0 for c in srv.poll())
    same(np.concatenate([b.download(meso.HIT_DTYPE, 41 * 27) for b in bufs]), 6)


def test_a_far_view_does_not_step_through_empty_bricks(ctx):
    # 1,900 voxels of sky above the ground, looked through from just within and
    # just beyond what the region walk takes: 237 bricks in four cubes
    scene = ctx.scene_from_terrain(meso.Terrain(512, 512, 2048, 3, 256, 6, 56.0, 60.0, 48, 0.7))
    out = ctx.alloc(24 * 1280 * 720)

    def us(z):
        cam = meso.camera((250.0, 240.0, z), (256.0, 256.0, 0.0), 1280, 720)
        cam.tan_half_fov_y = 140.0 / z
        a, b, best = ctx.event(), ctx.event(), float("inf")
        for _ in range(12):
            ctx.record(a)
            ctx.raymarch(scene, cam, shadow=False, out=out, download=False)
            ctx.record(b)
            best = min(best, 1e3 * ctx.elapsed_ms(a, b))
        return best

    near, far = us(120000.0), us(140000.0)
    print(f"near {near:.1f} us, far {far:.1f} us")
    assert far < 2.5 * near
    scene.destroy()
