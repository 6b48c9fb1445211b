"""What scenes take of the device's memory and when they give it back, on a CUDA runtime of host memory."""
import ctypes

import pytest

import mesoengine_gb300 as meso
import host_runtime

KEPT = 1 << 30  # of freed scenes' memory, by a context


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return host_runtime.load(tmp_path_factory.mktemp("host"))


@pytest.fixture
def path(tmp_path):
    return host_runtime.scene_file(tmp_path / "s", (64, 32, 96), 90)


def load(lib, ctx, path, spare):
    scene = ctypes.c_void_p()
    rc = lib.meso_scene_load(ctx, path, spare, ctypes.byref(scene))
    return rc, scene


@pytest.mark.parametrize("spare", [0, 900_000, 1_100_000, 3_000_000])  # up to and beyond what is kept
def test_a_destroyed_scene_is_given_back(lib, path, spare):
    ctx = host_runtime.context(lib)
    before = lib.fake_taken()
    rc, first = load(lib, ctx, path, spare)
    rc2, second = load(lib, ctx, path, spare // 2)
    assert rc == rc2 == 0 and lib.fake_taken() - before > 1500 * spare
    lib.meso_scene_destroy(ctx, first)
    assert lib.fake_taken() - before <= 1200 * (spare // 2) + (1 << 20) + KEPT
    lib.meso_scene_destroy(ctx, second)
    assert lib.fake_taken() - before <= KEPT
    lib.meso_ctx_destroy(ctx)


@pytest.mark.parametrize("dims,n,spare", [((32, 32, 32), 0, 0), ((64, 32, 96), 90, 0), ((64, 32, 96), 90, 5000),
                                          ((512, 256, 1024), 0, 0)])  # nothing but a pointer grid and its maps
def test_budgets_count_what_a_scene_takes(lib, tmp_path, dims, n, spare):
    path = host_runtime.scene_file(tmp_path / "s", dims, n)
    ctx = host_runtime.context(lib)
    before = lib.fake_live_bytes()
    rc, scene = load(lib, ctx, path, spare)
    info = meso.SceneInfo()
    assert rc == 0 and lib.meso_scene_get_info(ctx, scene, ctypes.byref(info)) == 0
    takes = lib.fake_live_bytes() - before
    assert info.device_bytes == takes
    lib.meso_scene_destroy(ctx, scene)
    lib.meso_ctx_destroy(ctx)
    for budget, status in ((takes - 1, 3), (takes, 0), (2 * takes - 1, 0), (2 * takes, 0)):
        ctx = host_runtime.context(lib, budget)
        rc, first = load(lib, ctx, path, spare)
        assert rc == status
        if rc == 0:
            rc, second = load(lib, ctx, path, spare)
            assert rc == (0 if budget == 2 * takes else 3)
            lib.meso_scene_destroy(ctx, first)
            if rc == 0:
                lib.meso_scene_destroy(ctx, second)
            rc, first = load(lib, ctx, path, spare)  # what was charged is given back
            assert rc == 0
            lib.meso_scene_destroy(ctx, first)
        lib.meso_ctx_destroy(ctx)


def test_small_scenes_follow_one_another_without_a_wait(lib, path):
    # a scene made in place of another finds the memory of the last one
    ctx = host_runtime.context(lib)
    rc, scene = load(lib, ctx, path, 100_000)
    held = lib.fake_taken()
    lib.fake_clear_log()
    lib.meso_scene_destroy(ctx, scene)
    calls = host_runtime.log(lib)
    last = max(i for i, c in enumerate(calls) if c[0] == "free")
    assert lib.fake_taken() == held and not [c for c in calls[last:] if c[0].startswith("wait")]
    rc, scene = load(lib, ctx, path, 100_000)
    assert rc == 0 and lib.fake_taken() == held
    lib.meso_scene_destroy(ctx, scene)
    lib.meso_ctx_destroy(ctx)


def test_a_scene_that_does_not_fit_is_given_back(lib, path):
    # the occupancy of 30 M slots (1.9 GB) fits, the materials do not
    ctx = host_runtime.context(lib)
    before = lib.fake_taken()
    lib.fake_limit(before + (8 << 30))
    rc, scene = load(lib, ctx, path, 30_000_000)
    lib.fake_limit(0)
    assert rc == 2 and not scene.value
    assert lib.fake_taken() - before <= KEPT
    lib.meso_ctx_destroy(ctx)


def full_device(lib, path):
    """A context that keeps 0.5 GB of a destroyed scene on a device with 64 MB to spare, and a small live scene."""
    ctx = host_runtime.context(lib)
    _, kept = load(lib, ctx, path, 500_000)
    _, scene = load(lib, ctx, path, 0)
    lib.meso_scene_destroy(ctx, kept)
    lib.fake_limit(lib.fake_taken() + (64 << 20))
    return ctx, scene


def dev_alloc(lib, ctx, scene, n):
    p = ctypes.c_void_p()
    rc = lib.meso_dev_alloc(ctx, n, ctypes.byref(p))
    return rc, lambda: lib.meso_dev_free(ctx, p)


def server(lib, ctx, scene, n):
    cfg, h = meso.ServerConfig(), ctypes.c_void_p()
    cfg.max_inflight_batches, cfg.max_batch_rays, cfg.max_edit_quads = 1, n // 24, 1024
    rc = lib.meso_server_create(ctx, ctypes.byref(cfg), (ctypes.c_void_p * 1)(scene), 1, ctypes.byref(h))
    return rc, lambda: lib.meso_server_destroy(h)


def mesh(lib, ctx, scene, n):
    # a temporary of the call: the quads of one chunk of host memory
    chunk, total = (ctypes.c_uint16 * 32768)(), ctypes.c_uint64()
    return lib.meso_mesh_host(ctx, 1, chunk, 1, 0, 0, None, 1, None, n // 8, ctypes.byref(total)), lambda: None


@pytest.mark.parametrize("take", [dev_alloc, server, mesh])
def test_kept_memory_goes_back_before_an_allocation_fails(lib, path, take):
    ctx, scene = full_device(lib, path)
    rc, give = take(lib, ctx, scene, 400 << 20)
    assert rc == 0
    give()
    rc, _ = take(lib, ctx, scene, 900 << 20)  # more than there is
    lib.fake_limit(0)
    assert rc == 2
    lib.meso_scene_destroy(ctx, scene)
    lib.meso_ctx_destroy(ctx)
