"""Loading a scene file: the order of its copies and its kernels, on a CUDA runtime of host memory.

A copy from pageable memory on the default stream may return before its data has
reached the device, and the context's stream does not wait for that stream: the
maps' kernels would read what the arrays held before.
"""
import ctypes

import pytest

import host_runtime


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return host_runtime.load(tmp_path_factory.mktemp("host"))


def load(lib, ctx, path, spare=7):
    lib.fake_clear_log()
    scene = ctypes.c_void_p()
    rc = lib.meso_scene_load(ctx, path, spare, ctypes.byref(scene))
    return rc, scene, host_runtime.log(lib)


@pytest.mark.parametrize("dims,n", [((32, 32, 32), 0), ((32, 32, 32), 64), ((96, 64, 160), 700)])
def test_kernels_come_after_the_copies_they_read(lib, tmp_path, dims, n):
    ctx = host_runtime.context(lib)
    rc, scene, calls = load(lib, ctx, host_runtime.scene_file(tmp_path / "s", dims, n))
    assert rc == 0
    copied = set()  # streams with copies that nothing has waited for
    uploads = launches = 0
    for c in calls:
        if c[0] in ("copy", "copy_and_return") and c[1] == "h2d":
            copied.add(c[2])
            uploads += 1
        elif c[0] == "wait":
            copied.discard(c[1])
        elif c[0] == "wait_device":
            copied.clear()
        elif c[0] == "launch":
            assert copied <= {c[1]}, f"{c[2]} on stream {c[1]} may run before copies on {copied}"
            launches += 1
    assert uploads == (4 if n else 2) and launches == (3 if n else 2)
    assert not copied  # the file's contents are given up when the call returns
    lib.meso_scene_destroy(ctx, scene)
    lib.meso_ctx_destroy(ctx)


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_a_failing_copy_leaves_nothing_in_flight(lib, tmp_path, k):
    ctx = host_runtime.context(lib)
    before = lib.fake_live_bytes()
    path = host_runtime.scene_file(tmp_path / "s", (64, 32, 32), 100)
    lib.fake_fail_copy(k)
    rc, scene, calls = load(lib, ctx, path)
    assert rc == 6 and not scene.value
    assert lib.fake_live_bytes() == before
    copies = [i for i, c in enumerate(calls) if c[0] == "copy"]
    frees = [i for i, c in enumerate(calls) if c[0] == "free"]
    # the copies that were issued have ended before the file's contents and the arrays go
    assert copies and any(calls[i] == ["wait", calls[copies[-1]][2]] for i in range(copies[-1], frees[0]))
    lib.meso_ctx_destroy(ctx)
