"""The mesher's word-wide greedy sweep and its emission against the oracle.

Patterns that reach the limits of the 32-bit row words: quads of every width
and height up to 32, rows of 16 unit quads, quads that end together, neighbours
in the same material that must not merge, materials that differ in one bit, and
words with one, a few and many quads, for 16-bit and 8-bit sources with and
without neighbouring chunks.
"""
import numpy as np
import pytest

import mesoengine_gb300 as meso
import oracle

pytestmark = pytest.mark.gpu


def runs(rng, axis, materials, empty):
    """Runs of random lengths 1..32 along one axis, alike along another."""
    a = np.zeros((32, 32, 32), dtype=np.uint16)
    for i in range(32):
        for j in range(32):
            k = 0
            while k < 32:
                n = int(rng.integers(1, 33))
                a[i, j, k:k + n] = 0 if rng.random() < empty else rng.choice(materials)
                k += n
        if rng.random() < 0.7:  # the next plane the same: tall quads
            a[i] = a[max(i - 1, 0)]
    return np.moveaxis(a, 2, axis)


def chunks():
    rng = np.random.default_rng(11)
    x, y, z = np.meshgrid(np.arange(32), np.arange(32), np.arange(32), indexing="ij")
    out = [np.ones((32, 32, 32)), (x + y + z) % 2 * 7, (x + y) % 2 * 200, x % 2 + 1, y % 3, (z % 5 == 0) * 9,
           (x == 31) & (y == 0), (x * y * z == 31 ** 3) * 1, 1 + (x // 8 + y // 8 + z // 8) % 2 * 127]
    for axis in range(3):
        for empty in (0.05, 0.4, 0.9):
            out.append(runs(rng, axis, [1, 2, 128, 129], empty))
    for p in (0.0005, 0.01, 0.1, 0.5, 0.97):
        out.append((rng.random((32, 32, 32)) < p) * rng.integers(1, 3, (32, 32, 32)))
        out.append((rng.random((32, 32, 32)) < p) * rng.integers(1, 256, (32, 32, 32)))
    return np.stack(out).astype(np.uint16)


CH = chunks()


@pytest.mark.parametrize("wide", [False, True])
def test_chunk_arrays(ctx, wide):
    # wide: 16-bit materials that differ in high or low bits only
    data = np.where(CH > 0, CH * 257 % 65535 + 1, 0).astype(np.uint16) if wide else CH.astype(np.uint8)
    kind = meso.SRC_CHUNKS_U16 if wide else meso.SRC_CHUNKS_U8
    ok = oracle.SRC_CHUNKS_U16 if wide else oracle.SRC_CHUNKS_U8
    ref = oracle.mesh_chunks(ok, data)
    d = ctx.to_device(data)
    for per_launch in (False, True):
        q, counts = ctx.mesh(kind, d, n=len(data), chunk_counts=True, per_launch=per_launch)
        assert np.array_equal(np.sort(q), ref)
        assert np.array_equal(counts, np.bincount((ref >> np.uint64(44)).astype(np.int64), minlength=len(data)))


@pytest.mark.parametrize("n", [1, 2, 40, 1300])
def test_lists_of_every_length(ctx, n):
    # from one chunk to several per block, in any order and repeated
    rng = np.random.default_rng(n)
    index = rng.integers(0, len(CH), n).astype(np.int32)
    q, _ = ctx.mesh(meso.SRC_CHUNKS_U16, ctx.to_device(CH), coords=index, n=n, capacity=n * 30000 + 98304)
    one = oracle.mesh_chunks(oracle.SRC_CHUNKS_U16, CH)
    chunk, low = (one >> np.uint64(44)).astype(np.int64), one & np.uint64((1 << 44) - 1)
    ref = np.concatenate([low[chunk == c] | np.uint64(k << 44) for k, c in enumerate(index)])
    assert np.array_equal(np.sort(q), ref)


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_neighbouring_chunks(ctx, dtype):
    # all patterns side by side in a grid and as a brick map: faces between
    # chunks are hidden by the neighbour
    g = np.zeros((96, 96, 96), dtype=dtype)
    for k in range(27):
        a, b, c = k // 9 * 32, k // 3 % 3 * 32, k % 3 * 32
        g[a:a + 32, b:b + 32, c:c + 32] = CH[k % len(CH)]
    coords = np.array([(x, y, z) for z in range(3) for y in range(3) for x in range(3)], dtype=np.int32)
    kind, ok = ((meso.SRC_GRID_U8, oracle.SRC_GRID_U8) if dtype == np.uint8 else (meso.SRC_GRID_U16, oracle.SRC_GRID_U16))
    ref = oracle.mesh_chunks(ok, g, coords=coords)
    q, _ = ctx.mesh(kind, ctx.to_device(g), coords=coords, dims=(96, 96, 96))
    assert np.array_equal(np.sort(q), ref)
    scene = ctx.scene_from_dense(g.astype(np.uint16))
    q, _ = ctx.mesh(meso.SRC_BRICKMAP, coords=coords, scene=scene)
    assert np.array_equal(np.sort(q), ref)
    scene.destroy()


@pytest.mark.parametrize("n", [1, 303, 305, 2431, 2432, 4864, 4871])
def test_lists_around_the_ticket_sizes(ctx, n):
    # entries per ticket change with the list's length; every entry is meshed
    # once, air chunks and chunks that the list names again among them
    g = np.zeros((64, 96, 96), dtype=np.uint16)
    g[:32, 32:64, 64:96] = CH[9 % len(CH)]
    g[32:40, 5, :50] = 3
    scene = ctx.scene_from_dense(g)
    every = np.array([(x, y, z) for z in range(2) for y in range(3) for x in range(3)], dtype=np.int32)
    ref = [oracle.mesh_chunks(oracle.SRC_GRID_U16, g, coords=every[k:k + 1]) for k in range(len(every))]
    coords = np.resize(every, (n, 3))
    q, _ = ctx.mesh(meso.SRC_BRICKMAP, coords=coords, scene=scene)
    want = np.concatenate([ref[k % len(every)] | np.uint64(k << 44) for k in range(n)])
    assert np.array_equal(np.sort(q), np.sort(want))
    scene.destroy()
