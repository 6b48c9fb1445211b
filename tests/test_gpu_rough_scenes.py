"""Scenes of scattered voxels: their rays walk step by step, with the same hits, and no slower than so.

Where little of the space is empty a block, the region walk leaves region after
region of one voxel.  A build counts the blocks and gives such a scene's views to the
walk that steps; scenes on both sides of the rule, from every kind of build, have to
give the oracle's bytes, alone and beside scenes of the other kind.
"""
import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


def scattered(dims, share, seed=1):
    rng = np.random.default_rng(seed)
    g = (rng.random(dims[::-1], dtype=np.float32) < share).astype(np.uint16)
    return g * rng.integers(1, 256, g.shape, dtype=np.uint16)


def same(got, ref):
    bad = np.nonzero((got.view(np.uint8).reshape(-1, 24) != ref.view(np.uint8).reshape(-1, 24)).any(1))[0]
    assert bad.size == 0, f"{bad.size} of {got.size} hits differ, first {got[bad[:3]]} vs {ref[bad[:3]]}"


@pytest.mark.parametrize("share", [0.0, 0.01, 0.03, 0.04, 0.1, 0.25, 0.6, 0.97, 1.0])
@pytest.mark.parametrize("build", ["dense", "grid_u8", "load"])
def test_hits(ctx, share, build, tmp_path):
    dims = (96, 64, 160)
    g = scattered(dims, share)
    bm = oracle.HostBrickMap.from_dense(g)
    if build == "grid_u8":
        scene = ctx.scene_from_grid(meso.SRC_GRID_U8, ctx.to_device(g.astype(np.uint8)), dims)
    else:
        scene = ctx.scene_from_dense(g)
    if build == "load":
        scene.save(str(tmp_path / "s"))
        scene.destroy()
        scene = ctx.scene_load(str(tmp_path / "s"))
    poses = [((-31.0, -17.0, 190.0), (48.0, 32.0, 80.0)), ((130.0, 90.0, -20.0), (40.0, 30.0, 90.0)),
             ((48.3, 32.2, 80.4), (90.0, 40.0, 20.0)), ((48.0, 32.0, 200.0), (48.0, 32.0, 0.0))]
    for shadow in (False, True):
        for o, t in poses:
            same(ctx.raymarch(scene, meso.camera(o, t, 65, 43), shadow=shadow),
                 oracle.raymarch(bm, oracle.camera(o, t, 65, 43), shadow=shadow))
    scene.destroy()


@pytest.mark.parametrize("n", [2, 5, 40])
def test_both_kinds_in_one_launch(ctx, n):
    dims = (96, 64, 160)
    grids = [scattered(dims, 0.2), scattered(dims, 0.002)]
    scenes = [ctx.scene_from_dense(g) for g in grids]
    maps = [oracle.HostBrickMap.from_dense(g) for g in grids]
    poses = [(-31.0, -17.0, 190.0), (130.0, 90.0, -20.0), (48.3, 32.2, 80.4)]
    for pick in ([k % 2 for k in range(n)], [0] * n):  # both, and only the rough one
        cams = [(poses[k % 3], (40.0, 33.0, 70.0), 33 + k, 21) for k in range(n)]
        ref = np.concatenate([oracle.raymarch(maps[s], oracle.camera(*c)) for s, c in zip(pick, cams)])
        same(ctx.raymarch([scenes[s] for s in pick], [meso.camera(*c) for c in cams]), ref)
        srv = meso.Server(ctx, scenes, max_inflight_batches=1, max_batch_rays=1 << 20)
        bufs = [ctx.alloc(24 * c[2] * c[3]) for c in cams]
        for k, c in enumerate(cams):
            srv.submit(pick[k], meso.camera(*c), shadow=True, tag=k, dst=bufs[k])
        srv.drain(20.0)
        done = srv.poll()
        assert len(done) == n and all(d.status == 0 for d in done)
        same(np.concatenate([b.download(meso.HIT_DTYPE, c[2] * c[3]) for b, c in zip(bufs, cams)]), ref)
        del srv
    for s in scenes:
        s.destroy()


@pytest.mark.parametrize("share", [0.1, 0.25])
def test_scattered_voxels_are_walked_by_steps(ctx, share):
    # one view from just within what the region walk takes and one from just
    # beyond it, which steps: the same rays, all but for their origin
    scene = ctx.scene_from_dense(scattered((256, 256, 256), share))
    out = ctx.alloc(24 * 1920 * 1080)

    def us(z):
        cam = meso.camera((100.0 + 0.3 * z, 110.0 + 0.2 * z, z), (128.0, 128.0, 128.0), 1920, 1080)
        cam.tan_half_fov_y = 90.0 / z
        a, b, best = ctx.event(), ctx.event(), float("inf")
        for _ in range(15):
            ctx.record(a)
            ctx.raymarch(scene, cam, out=out, download=False)
            ctx.record(b)
            best = min(best, 1e3 * ctx.elapsed_ms(a, b))
        return best

    near, far = us(115000.0), us(140000.0)
    print(f"share {share}: near {near:.1f} us, far {far:.1f} us")
    assert near < 1.1 * far
    scene.destroy()
