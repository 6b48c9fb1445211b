"""The work that programs give this framework, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a program holds before the call (a context, scenes, inputs and output
buffers in device memory), `run` is one pass through the public entry points.  Sizes are those of the framework's own workloads
(bench.py, the terrain presets, the tests) and of ordinary programs around them; `draw` gives more of the same ranges.

Every output is a packed integer record (hits of 24 bytes, 64-bit quads, vertices, bit rows, brick pools), equal bit for bit from
run to run, so no case has a value in 64-bit floating point and there is no `exact`.
"""
import ctypes
import math

import numpy as np
import torch

import mesoengine_gb300 as meso

_ctx = None


def context():
    """One context for the process, as a program has."""
    global _ctx
    if _ctx is None:
        _ctx = meso.Context(0)
    return _ctx


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a thumbnail or a probe view of a small scene: one small launch, latency counts
        {"name": "view_256", "op": "view", "scene": "terrain", "n": 512, "w": 256, "h": 256, "views": 1, "shadow": False},
        # the small plain workload: a 640x360 view to the first hit over a dense 256^3 noise grid
        {"name": "view_noise_640x360", "op": "view", "scene": "noise", "n": 256, "w": 640, "h": 360, "views": 1, "shadow": False},
        # the headline frame: 1920x1080, primary and shadow rays, 1024^3 terrain, hits left on the device
        {"name": "frame_1080p_shadow", "op": "view", "scene": "terrain", "n": 1024, "w": 1920, "h": 1080, "views": 1, "shadow": True},
        # the same frame for a program that wants the hits in its page-locked host buffer
        {"name": "frame_1080p_host", "op": "host", "n": 1024, "w": 1920, "h": 1080, "shadow": True},
        # served rendering: a burst of requests over four resident scenes, 256^2 to 3840x2160, through the request server
        {"name": "serve_burst_40", "op": "serve", "n": 2048, "requests": 40, "max_w": 3840},
        # batched meshing: 4096 standalone uint16 chunks, occupancy log-uniform in 0.1..90 %
        {"name": "mesh_u16_4096", "op": "mesh", "kind": "chunks_u16", "chunks": 4096},
        # the dense 256^3 uint8 grid, all 512 chunks in one call
        {"name": "mesh_grid_u8_512", "op": "mesh", "kind": "grid_u8", "chunks": 512},
        # first meshing of a whole resident scene: every chunk of the 1024^3 terrain, four in five of them air
        {"name": "mesh_scene_32768", "op": "mesh", "kind": "scene", "chunks": 32768},
        # a raster consumer's refresh: the 180 chunks around some edits meshed again and expanded to vertices
        {"name": "remesh_vertices_180", "op": "vertices", "kind": "scene", "chunks": 180},
        # an edit as an interactive program makes it: 16 spheres, the resident mesh brought up to date, a 1080p view
        {"name": "edit_remesh_1080p", "op": "edit", "n": 2048, "spheres": 16, "w": 1920, "h": 1080},
        # a scene made from a dense grid already on the device, in place of the last one
        {"name": "build_grid_u16_512", "op": "build", "kind": "grid_u16", "nx": 512, "ny": 512, "nz": 512},
        # the reference's erosion pyramid of 4096 chunks, four levels
        {"name": "erode_u16_4096", "op": "erode", "kind": "chunks_u16", "chunks": 4096, "depth": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng, lo, hi):
    """A grid dimension: a multiple of 32."""
    return max(lo, min(hi, 32 * max(1, round(_log(rng, lo, hi) / 32))))


def _image(rng, most_w, most_h):
    """An image size, odd ones and widths off the 8-pixel tile among them."""
    return max(48, min(most_w, _log(rng, 48, most_w) | rng.choice((0, 1)))), max(32, min(most_h, _log(rng, 32, most_h) | rng.choice((0, 1))))


KINDS = ("chunks_u16", "chunks_u8", "grid_u8", "grid_u16", "scene")


def draw(rng):
    op = rng.choice(("view", "view", "host", "serve", "mesh", "mesh", "vertices", "edit", "build", "erode"))
    if op == "view":
        w, h = _image(rng, 3840, 2160)
        views = min(_log(rng, 1, 48), max(1, 12_000_000 // (w * h)))
        scene = rng.choice(("terrain", "terrain", "noise"))
        return {"op": op, "scene": scene, "n": _dim(rng, 96, 512 if scene == "noise" else 1024), "w": w, "h": h, "views": views,
                "shadow": rng.random() < 0.5}
    if op == "host":
        w, h = _image(rng, 3840, 2160)
        return {"op": op, "n": _dim(rng, 128, 1024), "w": w, "h": h, "shadow": rng.random() < 0.5}
    if op == "serve":
        return {"op": op, "n": _dim(rng, 256, 1024), "requests": _log(rng, 2, 40), "max_w": rng.choice((256, 512, 1920, 3840))}
    if op in ("mesh", "vertices", "erode"):
        case = {"op": op, "kind": rng.choice(KINDS), "chunks": _log(rng, 1, 4096 if op != "vertices" else 512)}
        if op == "erode":
            case["depth"] = rng.randint(1, 8)
        return case
    if op == "edit":
        w, h = _image(rng, 1920, 1080)
        return {"op": op, "n": _dim(rng, 256, 2048), "spheres": rng.randint(1, 32), "w": w, "h": h}
    return {"op": op, "kind": rng.choice(("grid_u8", "grid_u16")), "nx": _dim(rng, 64, 512), "ny": _dim(rng, 64, 512),
            "nz": _dim(rng, 64, 512)}


# ------------------------------------------------------------------ inputs

def _terrain(n, seed):
    """The presets' recipe (bench scene: period n/2, amplitude n/4, about 15 % solid) at n^3."""
    return meso.Terrain(n, n, n, seed & 0x7FFFFFFF, max(1, n // 2), 6, 56.0 * n / 1024.0, n / 4.0, 48, 0.7)


def _frame_camera(n, w, h, rng):
    """The bench's view of the scene, from a spot near its own."""
    o = (np.array([-300.0, -200.0, 800.0]) + rng.uniform(-16, 16, 3)) * (n / 1024.0)
    return meso.camera(o, (n / 2.0, n / 2.0, n / 2.0), w, h)


def _outside_camera(n, w, h, rng):
    """A random pose outside the scene, looking at the ground (the served streams' poses)."""
    v = rng.normal(size=3)
    v[2] = abs(v[2]) + 0.2
    v /= np.linalg.norm(v)
    return meso.camera(np.full(3, n / 2.0) + v * 1.1 * n,
                       (rng.uniform(0.25, 0.75) * n, rng.uniform(0.25, 0.75) * n, rng.uniform(0.02, 0.2) * n), w, h)


class _Raw:
    """Device memory of the framework, as torch sees it (no copy)."""

    def __init__(self, ptr, n, typestr, keep=None):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (int(ptr), False), "version": 3}


def _tensor(ptr, n, typestr="<i8", keep=None):
    if n == 0:
        return torch.zeros(0, dtype=torch.int64, device="cuda")
    return torch.as_tensor(_Raw(ptr, n, typestr, keep), device="cuda")


class Outputs(tuple):
    """What a pass leaves in the program's buffers, read where it is looked at.

    The mesher appends quads in the order in which its blocks finish, so a quad list is a set: it is read here in numeric order of
    the packed words (chunk, direction, z, y, x).  A program draws or stores the quads as they lie, so the ordering, which serves
    only to compare two passes, is no part of one."""

    def __new__(cls, read):
        self = super().__new__(cls)
        self.read = read
        return self

    def __iter__(self):
        return iter(self.read())


def _u8_grid(n3, seed):
    """The noise grid of the small plain workload, nx x ny x nz."""
    return context().generate_dense_u8(n3[0], n3[1], n3[2], seed=seed & 0x7FFFFFFF)


def _u16_of(buf, count):
    """A uint16 copy of a uint8 buffer's materials, spread over more than 8 bits."""
    v = _tensor(buf.ptr, count, "|u1", buf).to(torch.int16)
    v = torch.where(v > 0, v * 37 + 300, v)
    out = context().alloc(2 * count)
    _tensor(out.ptr, count, "<i2", out).copy_(v)
    torch.cuda.synchronize()
    return out


def _chunk_grid(chunks):
    """The dims of a dense grid of at least `chunks` chunks."""
    e = max(1, round(chunks ** (1 / 3)))
    ez = -(-chunks // (e * e))
    return (32 * e, 32 * e, 32 * ez)


def _source(case, seed):
    """(MeshSource, coordinate buffer or None, what they keep alive) of a meshing or erosion case."""
    ctx, kind, n = context(), case["kind"], case["chunks"]
    src = meso.MeshSource()
    if kind in ("chunks_u16", "chunks_u8"):
        data, _ = ctx.generate_chunks_u16(n, seed0=seed & 0x3FFFFFFF)
        if kind == "chunks_u8":
            wide = _tensor(data.ptr, n * 32768, "<i2", data)
            data = ctx.alloc(n * 32768)
            _tensor(data.ptr, n * 32768, "|u1", data).copy_(wide.to(torch.uint8))
            torch.cuda.synchronize()
        src.kind = meso.SRC_CHUNKS_U16 if kind == "chunks_u16" else meso.SRC_CHUNKS_U8
        src.d_data = data.ptr
        return src, None, data
    if kind in ("grid_u8", "grid_u16"):
        dims = _chunk_grid(n)
        data = _u8_grid(dims, seed)
        if kind == "grid_u16":
            data = _u16_of(data, dims[0] * dims[1] * dims[2])
        src.kind = meso.SRC_GRID_U8 if kind == "grid_u8" else meso.SRC_GRID_U16
        src.d_data = data.ptr
        src.nx, src.ny, src.nz = dims
        e, k = dims[0] // 32, np.arange(n)
        xyz = np.stack([k % e, (k // e) % e, k // (e * e)], 1)
    else:
        data = ctx.scene_from_terrain(_terrain(1024, seed))  # 32 x 32 x 32 chunks
        src.kind, src.scene = meso.SRC_BRICKMAP, data.handle
        if n == 32768:
            k = np.arange(n)
        else:  # the chunks around the ground, as edits leave them
            rng = np.random.default_rng(seed)
            hill = rng.integers(0, 1024, size=max(1, n // 8))
            k = (hill[:, None] + np.array([0, 1, 32, 33, 1024, 1025, 1056, 1057])[None, :]).reshape(-1)
            k = k + 1024 * rng.integers(1, 6, size=k.size)
            k = np.resize(np.unique(np.minimum(k, 32767)), n)
        xyz = np.stack([k % 32, (k // 32) % 32, k // 1024], 1)
    coords = ctx.to_device(np.ascontiguousarray(xyz, dtype=np.int32))
    return src, coords, data


def _quad_room(case):
    """A quad buffer that holds any list of up to 256 chunks, and a generous share per chunk beyond."""
    n = case["chunks"]
    return n * 98304 if n <= 256 else max(256 * 98304, n * (8192 if n <= 4096 else 1024))


def _whole(v, n, size):
    """The n first values of v, and zeros up to a size that is the same for all inputs of a case."""
    out = torch.zeros((size,) + v.shape[1:], dtype=v.dtype, device=v.device)
    out[:n] = v[:n]
    return out


def prepare(case, seed):
    ctx, op, rng = context(), case["op"], np.random.default_rng(seed)
    s = {"op": op, "ctx": ctx, "case": dict(case)}
    if op in ("view", "host"):
        n = case["n"]
        if case.get("scene") == "noise":
            grid = _u8_grid((n, n, n), seed)
            s["scene"] = ctx.scene_from_grid(meso.SRC_GRID_U8, grid, (n, n, n))
            o = (np.array([-0.35, -0.25, 0.9]) + rng.uniform(-0.02, 0.02, 3)) * n
            cams = [meso.camera(o, (n / 2.0,) * 3, case["w"], case["h"])]
        else:
            s["scene"] = ctx.scene_from_terrain(_terrain(n, seed))
            cams = [_frame_camera(n, case["w"], case["h"], rng)]
        cams += [_outside_camera(n, case["w"], case["h"], rng) for _ in range(case.get("views", 1) - 1)]
        s["cams"], s["shadow"] = cams, case["shadow"]
        words = 3 * sum(c.width * c.height for c in cams)
        s["out"] = ctx.alloc(8 * words) if op == "view" else ctx.pinned(8 * words)
        s["hits"] = _tensor(s["out"].ptr, words, keep=s["out"]) if op == "view" else s["out"].view(np.int64, words)
    elif op == "serve":
        n = case["n"]
        sides = (n // 4 // 32 * 32, n // 2 // 32 * 32, n // 2 // 32 * 32, n)
        s["scenes"] = [ctx.scene_from_terrain(_terrain(e, seed + 17 * k)) for k, e in enumerate(sides)]
        s["server"] = meso.Server(ctx, s["scenes"], max_inflight_batches=4, max_batch_rays=16 << 20, hbm_budget_bytes=120 << 30)
        sizes = [z for z in ((256, 256), (512, 512), (1920, 1080), (3840, 2160)) if z[0] <= case["max_w"]]
        s["requests"], s["hits"] = [], []
        for k in range(case["requests"]):
            i, (w, h) = int(rng.integers(0, 4)), sizes[k % len(sizes)]
            dst = ctx.alloc(24 * w * h)
            s["requests"].append((i, _outside_camera(sides[i], w, h, rng), dst))
            s["hits"].append(_tensor(dst.ptr, 3 * w * h, keep=dst))
    elif op in ("mesh", "vertices"):
        s["src"], s["coords"], s["data"] = _source(case, seed)
        room, n = _quad_room(case), case["chunks"]
        s["quads"], s["count"], s["counts"] = ctx.alloc(8 * room), ctx.alloc(8), ctx.alloc(4 * n)
        s["mesh_out"] = meso.MeshOutput(s["quads"].ptr, room, s["count"].ptr, s["counts"].ptr)
        s["t"] = (_tensor(s["quads"].ptr, room), _tensor(s["count"].ptr, 1), _tensor(s["counts"].ptr, n, "<i4"))
        if op == "vertices":
            s["origins"] = ctx.to_device(np.stack([np.arange(n) % 64, np.arange(n) // 64, np.zeros(n)], 1).astype(np.int32))
            s["room"] = 4 * n * CHUNK_QUADS[case["kind"]] + 4 * 98304
            s["verts"] = ctx.alloc(64 * s["room"])
            s["tv"] = _tensor(s["verts"].ptr, 16 * s["room"], "<i4", s["verts"])
    elif op == "edit":
        n = case["n"]
        s["scene"] = ctx.scene_from_terrain(_terrain(n, seed), spare_bricks=1 << 18)
        s["store"] = ctx.mesh_store(s["scene"])
        top = max(33, int(0.28 * n))
        s["edits"] = [meso.SphereEdit((ctypes.c_int32 * 3)(int(rng.integers(0, n)), int(rng.integers(0, n)), int(rng.integers(0, top))),
                                      int(rng.integers(2, 33)), 0 if rng.random() < 0.5 else int(rng.integers(1, 65536)), 0)
                      for _ in range(case["spheres"])]
        s["cam"] = _frame_camera(n, case["w"], case["h"], rng)
        words = 3 * case["w"] * case["h"]
        s["out"] = ctx.alloc(8 * words)
        s["hits"] = _tensor(s["out"].ptr, words, keep=s["out"])
    elif op == "build":
        dims = (case["nx"], case["ny"], case["nz"])
        s["grid"] = _u8_grid(dims, seed)
        if case["kind"] == "grid_u16":
            s["grid"] = _u16_of(s["grid"], dims[0] * dims[1] * dims[2])
        s["kind"] = meso.SRC_GRID_U8 if case["kind"] == "grid_u8" else meso.SRC_GRID_U16
        s["dims"], s["scene"] = dims, None
    else:  # erode
        s["src"], s["coords"], s["data"] = _source(case, seed)
        words = case["chunks"] * case["depth"] * 1024
        s["out"] = ctx.alloc(4 * words)
        s["mips"] = _tensor(s["out"].ptr, words, "<i4", s["out"])
    return s


# ------------------------------------------------------------------ one pass

def _mesh(s):
    """One call of the batched mesher into the program's buffers."""
    meso._check(meso.load().meso_mesh_chunks(s["ctx"].handle, ctypes.byref(s["src"]), s["coords"].ptr if s["coords"] else None,
                                             s["case"]["chunks"], ctypes.byref(s["mesh_out"]), None))


def _sorted_quads(s):
    quads, count, counts = s["t"]
    n = int(count.item())
    return [count, counts, _whole(torch.sort(quads[:n]).values, n, quads.numel())]


def _vertices(s, total):
    quads, count, counts = s["t"]
    order = torch.sort(quads[:total]).indices
    return [count, counts, _whole(s["tv"][: 16 * total].view(total, 16)[order], total, s["room"])]


def _built(s):
    i = s["scene"].info()
    n, most = int(i.n_bricks), (i.nx // 8) * (i.ny // 8) * (i.nz // 8)
    return [n, _tensor(i.d_ptr, most, "<i4"), _whole(_tensor(i.d_occ, 8 * n), 8 * n, 8 * most),
            _whole(_tensor(i.d_mat, 512 * n, "<i2"), 512 * n, 512 * most)]


def _edited(s, dirty):
    quads = np.sort(s["store"].gather(dirty)).view(np.int64)
    n = s["case"]["n"] // 32
    return [_whole(torch.from_numpy(dirty.astype(np.int64)), dirty.size, n * n * n), s["hits"],
            _whole(torch.from_numpy(quads), quads.size, 1 << 22)]


def run(s):
    ctx, op = s["ctx"], s["op"]
    if op == "view":
        ctx.raymarch(s["scene"], s["cams"], shadow=s["shadow"], out=s["out"], download=False)
        return s["hits"]
    if op == "host":
        ctx.raymarch_host(s["scene"], s["cams"][0], shadow=s["shadow"], out_ptr=s["out"].ptr)
        return Outputs(lambda: [s["hits"]])
    if op == "serve":
        srv = s["server"]
        for k, (i, cam, dst) in enumerate(s["requests"]):
            srv.submit(i, cam, shadow=False, tag=k, dst=dst)
        srv.drain(60.0)
        done = sorted(srv.poll(), key=lambda c: c.user_tag)
        return s["hits"] + [np.array([c.hit_checksum for c in done], dtype=np.uint64).view(np.int64),
                            np.array([c.status for c in done], dtype=np.int32)]
    if op == "mesh":
        _mesh(s)
        return Outputs(lambda: _sorted_quads(s))
    if op == "vertices":
        _mesh(s)
        total = ctypes.c_uint64()
        meso._check(meso.load().meso_mesh_check(ctx.handle, ctypes.byref(s["mesh_out"]), None, ctypes.byref(total)))
        n = min(int(total.value), s["room"])
        meso._check(meso.load().meso_quads_to_vertices(ctx.handle, s["quads"].ptr, n, s["origins"].ptr, s["case"]["chunks"],
                                                       s["verts"].ptr, None))
        return Outputs(lambda: _vertices(s, n))
    if op == "edit":
        dirty = s["scene"].edit(s["edits"])
        s["store"].update(dirty)
        ctx.raymarch(s["scene"], s["cam"], shadow=False, out=s["out"], download=False)
        return Outputs(lambda: _edited(s, dirty))
    if op == "build":
        s["scene"] = None  # the last scene goes before the next is made
        s["scene"] = ctx.scene_from_grid(s["kind"], s["grid"], s["dims"])
        return Outputs(lambda: _built(s))
    meso._check(meso.load().meso_erode_mips(ctx.handle, ctypes.byref(s["src"]), s["coords"].ptr if s["coords"] else None,
                                            s["case"]["chunks"], s["case"]["depth"], s["out"].ptr, None))
    return s["mips"]


# ------------------------------------------------------------------ what a pass cannot do without

CHUNK_BYTES = {"chunks_u16": 65536, "chunks_u8": 32768, "grid_u8": 32768, "grid_u16": 65536,
               # a chunk of the terrain: 64 pointers, and 16.8 % of its bricks (1 KiB of materials, 64 B of occupancy)
               "scene": 256 + 0.168 * 64 * 1088}
# quads of a chunk, on average over the generators' chunks (a scene's around the ground; over all of it 48)
CHUNK_QUADS = {"chunks_u16": 2780, "chunks_u8": 2780, "grid_u8": 540, "grid_u16": 540, "scene": 260}


def work(case):
    """Inputs read once and outputs written once.  A view's input is what its rays see: about one 8^3 brick's mask (64 B) and pointer
    for each 16 pixels, and a material for each pixel."""
    op = case["op"]
    if op in ("view", "host", "edit"):
        px = case["w"] * case["h"] * case.get("views", 1)
        b = px * (24 + 2 + 68 / 16)
        if op == "edit":  # each sphere: its box's bricks read and written, then its chunks meshed
            b += case["spheres"] * (100 * 2 * 1088 + 8 * (CHUNK_BYTES["scene"] + 8 * CHUNK_QUADS["scene"]))
        return {"bytes": b, "flops": 0}
    if op == "serve":
        sizes = [z for z in ((256, 256), (512, 512), (1920, 1080), (3840, 2160)) if z[0] <= case["max_w"]]
        return {"bytes": sum(sizes[k % len(sizes)][0] * sizes[k % len(sizes)][1] * (24 + 2 + 68 / 16) for k in range(case["requests"])), "flops": 0}
    if op in ("mesh", "vertices"):
        n, kind = case["chunks"], case["kind"]
        quads = n * (48 if kind == "scene" and n == 32768 else CHUNK_QUADS[kind])
        return {"bytes": n * CHUNK_BYTES[kind] + quads * (8 if op == "mesh" else 8 + 72), "flops": 0}
    if op == "build":
        vox = case["nx"] * case["ny"] * case["nz"]
        # the grid read, then a pointer, and for the bricks that hold anything (three in five of this noise's) their materials and masks
        return {"bytes": vox * (1 if case["kind"] == "grid_u8" else 2) + vox / 512 * (4 + 0.62 * 1088), "flops": 0}
    return {"bytes": case["chunks"] * (CHUNK_BYTES[case["kind"]] + 4096 * case["depth"]), "flops": 0}
