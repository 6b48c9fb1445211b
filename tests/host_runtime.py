"""The library's host code on a CUDA runtime made of host memory (cpp/fake_cudart.cpp).

Which call goes to which stream, what is waited for, how much memory is taken,
and what happens after a failing call can be seen there, without a GPU; kernels
do nothing, so results can not.
"""
import ctypes
import glob
import os
import struct
import subprocess

import mesoengine_gb300 as meso

HERE = os.path.dirname(os.path.abspath(__file__))


def load(folder):
    """A fresh copy of the library on the fake runtime, built in `folder`."""
    meso._build.build()
    out = os.path.join(str(folder), "libmeso_host.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    objects = sorted(glob.glob(os.path.join(os.path.dirname(meso.LIB_PATH), "*.o")))
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-O1", "-Wall", "-I", cuda, "-Wl,-Bsymbolic", "-Wl,-z,defs",
                    os.path.join(HERE, "cpp", "fake_cudart.cpp"), *objects, "-o", out, "-lpthread"], check=True)
    lib = ctypes.CDLL(out)
    for name, args in meso._SIGNATURES.items():
        fn = getattr(lib, name, None)
        if fn is not None:
            fn.argtypes = args
    lib.meso_last_error_string.restype = ctypes.c_char_p
    lib.fake_log.restype = lib.fake_taken.restype = lib.fake_live_bytes.restype = ctypes.c_size_t
    lib.fake_limit.argtypes = [ctypes.c_size_t]
    return lib


def log(lib):
    n = lib.fake_log(None, ctypes.c_size_t(0))
    buf = ctypes.create_string_buffer(n)
    lib.fake_log(buf, ctypes.c_size_t(n))
    return [line.split() for line in buf.value.decode().splitlines()]


def context(lib, budget=0):
    c, h = meso.Config(), ctypes.c_void_p()
    c.hbm_budget_bytes = budget
    assert lib.meso_ctx_create(ctypes.byref(c), ctypes.byref(h)) == 0
    return h


def scene_file(path, dims, n):
    """A scene file of `dims` voxels with its first n bricks occupied (one voxel each)."""
    nb = dims[0] * dims[1] * dims[2] // 512
    with open(path, "wb") as f:
        f.write(b"MESOBRK1" + struct.pack("<IiiiQ", 1, *dims, n))
        f.write(struct.pack(f"<{nb}I", *range(n), *[0xFFFFFFFF] * (nb - n)))
        f.write((struct.pack("<8Q", 1, *[0] * 7)) * n + struct.pack("<512H", 5, *[0] * 511) * n)
    return str(path).encode()
