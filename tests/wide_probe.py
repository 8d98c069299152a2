"""Builds and loads wide_probe.cu against the native library."""
import ctypes as C
import os
import subprocess

import numpy as np

from renderer2_b200 import _native  # noqa: F401 (the library it links with)
from renderer2_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))
SRC, LIB = os.path.join(HERE, "wide_probe.cu"), os.path.join(HERE, "_build", "libwideprobe.so")
_lib = None


def lib():
    global _lib
    if _lib is None:
        if B._needs(LIB, [SRC, B.LIB] + B._headers()):
            os.makedirs(os.path.dirname(LIB), exist_ok=True)
            r = subprocess.run([B.NVCC] + B.NVCC_FLAGS + ["-shared", "-cudart", "static", "-o", LIB, SRC, "-L", B.LIBDIR,
                                                          "-lrenderer2", "-Xlinker", "-rpath," + B.LIBDIR],
                               capture_output=True, text=True)
            assert r.returncode == 0, r.stderr
        _lib = C.CDLL(LIB)
        _lib.probe_wide_nodes.restype = C.c_uint64
        _lib.probe_wide_nodes.argtypes = [C.c_void_p, C.c_uint32, C.c_int, C.c_uint32, C.c_void_p]
        _lib.probe_tri_near.argtypes = [C.c_void_p] * 5 + [C.c_float, C.c_uint32, C.c_void_p]
        _lib.probe_tri_near.restype = None
        _lib.probe_trace.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p, C.c_uint32, C.c_void_p, C.c_uint32] + [C.c_void_p] * 5
    return _lib


def wide_nodes(boxes, skew, seed=1):
    """(wide nodes, capacity) of the collapse over leaf boxes, an (n, 6) array."""
    boxes = np.ascontiguousarray(boxes, np.float32)
    cap = C.c_uint64()
    n = lib().probe_wide_nodes(boxes.ctypes.data, boxes.shape[0], skew, seed, C.byref(cap))
    return n, cap.value


def trace(tris, rays):
    """Hits of the rays, an (n, 7) array of origin, direction and tmax, among (m, 3, 3) triangles: records (t, b1, b2,
    triangle) of the wide tree, of the binary one and of a test of every triangle, whether the wide any-hit query found
    one, and the wide nodes whose boxes the ray enters."""
    pos = np.ascontiguousarray(tris, np.float32).reshape(-1, 3)
    idx = np.arange(pos.shape[0], dtype=np.uint32)
    rays = np.ascontiguousarray(rays, np.float32)
    n = rays.shape[0]
    rec = np.dtype([("t", "<f4"), ("b1", "<f4"), ("b2", "<f4"), ("tri", "<i4")])
    a, b, c, seen, visits = (np.empty(n, t) for t in (rec, rec, rec, np.int32, np.uint32))
    status = lib().probe_trace(pos.ctypes.data, pos.shape[0], idx.ctypes.data, idx.size // 3, rays.ctypes.data, n,
                               a.ctypes.data, b.ctypes.data, c.ctypes.data, seen.ctypes.data,
                               visits.ctypes.data)
    assert status == 0, status
    for h in (a, b, c):
        h["t"][h["tri"] < 0] = 0.0
    return a, b, c, seen != 0, visits


def tri_near(tris, c0, around, c, r, voxel):
    """Whether the filter keeps each (n, 3, 3) triangle for the ball of radius r about c (test set up for centres within
    `around` of c0), among voxels of the given size."""
    a = [np.ascontiguousarray(x, np.float32) for x in (tris, c0, around, c, r)]
    near = np.empty(a[0].shape[0], np.int32)
    lib().probe_tri_near(*(x.ctypes.data for x in a), float(voxel), near.size, near.ctypes.data)
    return near != 0
