"""libhpt_bvhemu.so: the hierarchy's closest-hit query built for the host,
beside the tree walk (test infrastructure only)."""
import ctypes as C
import os
import subprocess

import numpy as np

from hptracing_b200._lib import SceneDesc

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
CSRC = os.path.join(ROOT, "hptracing_b200", "csrc")
LIB = os.path.join(HERE, "libhpt_bvhemu.so")
_lib = None


def build():
    srcs = [os.path.join(HERE, "bvh_emu.cu")] + [os.path.join(CSRC, f) for f in (
        "bvh_build.cpp", "scene_pack.cpp", "kdtree_build.cpp", "obj_loader.cpp")]
    deps = srcs + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    if os.path.exists(LIB) and os.path.getmtime(LIB) >= max(os.path.getmtime(x) for x in deps):
        return
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-fPIC,-ffp-contract=off,-pthread",
                        "-DHPT_DEVICE_CHECKS", "-I", os.path.join(ROOT, "include"), "-shared", "-o", LIB]
                       + srcs, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("bvhemu build failed\n%s%s" % (r.stdout, r.stderr))


def lib():
    global _lib
    if _lib is None:
        build()
        _lib = C.CDLL(LIB)
        _lib.bvhemu_create.restype = C.c_void_p
        _lib.bvhemu_create.argtypes = [C.POINTER(SceneDesc)]
        _lib.bvhemu_destroy.argtypes = [C.c_void_p]
        _lib.bvhemu_shape.argtypes = [C.c_void_p] * 2
        _lib.bvhemu_query.argtypes = [C.c_void_p, C.c_int] + [C.c_void_p] * 7
    return _lib


class BvhEmu:
    def __init__(self, mesh, nodes, leaf):
        d = SceneDesc()
        self._keep = [mesh.points, mesh.triangles, mesh.materials, nodes, leaf]
        d.points, d.num_points = mesh.points.ctypes.data, len(mesh.points)
        d.triangles, d.num_triangles = mesh.triangles.ctypes.data, len(mesh.triangles)
        d.materials, d.num_materials = mesh.materials.ctypes.data, len(mesh.materials)
        d.nodes, d.num_nodes = nodes.ctypes.data, len(nodes)
        d.leaf_data, d.num_leaf_data = leaf.ctypes.data, len(leaf)
        self.h = lib().bvhemu_create(C.byref(d))
        assert self.h

    def __del__(self):
        if getattr(self, "h", None):
            lib().bvhemu_destroy(self.h)

    def shape(self):
        c = np.zeros(3, np.int32)
        lib().bvhemu_shape(self.h, c.ctypes.data)
        return dict(nodes=int(c[0]), triangles=int(c[1]), depth=int(c[2]))

    def query(self, o, d):
        o, d = np.ascontiguousarray(o, np.float32), np.ascontiguousarray(d, np.float32)
        n = len(o)
        tri, walk_tri, certain = (np.zeros(n, np.int32) for _ in range(3))
        t, walk_t = np.zeros(n, np.float32), np.zeros(n, np.float32)
        flags = lib().bvhemu_query(self.h, n, *(x.ctypes.data for x in (o, d, tri, t, walk_tri, walk_t, certain)))
        return dict(tri=tri, t=t, walk_tri=walk_tri, walk_t=walk_t, certain=certain != 0, flags=flags)
