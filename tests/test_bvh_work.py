"""CPU test of how much a query through the hierarchy does: less than the tree
walk, also where its boxes have to be large."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import hptracing_b200 as H
from tests.test_bvh import _mesh, _scene, emu
from tests.test_bvh_bounds import _from_afar
from tests import scenes as S

LIB = os.path.join(emu.HERE, "libhpt_bvhwork.so")


def _work(mesh, nodes, leaf, o, d):
    """Node visits and tests of the query; node steps, leaves and tests of the walk."""
    emu.build()
    srcs = [os.path.join(emu.HERE, "bvh_work.cu")] + [os.path.join(emu.CSRC, f) for f in (
        "bvh_build.cpp", "scene_pack.cpp", "kdtree_build.cpp", "obj_loader.cpp")]
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(
            [os.path.getmtime(emu.LIB)] + [os.path.getmtime(s) for s in srcs]):
        subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-fPIC,-ffp-contract=off,-pthread",
                        "-DHPT_DEVICE_CHECKS", "-I", os.path.join(emu.ROOT, "include"), "-shared", "-o", LIB] + srcs,
                       check=True, capture_output=True)
    lib = C.CDLL(LIB)
    lib.bvhemu_create.restype = C.c_void_p
    lib.bvhemu_work.argtypes = [C.c_void_p, C.c_int] + [C.c_void_p] * 3
    lib.bvhemu_destroy.argtypes = [C.c_void_p]
    e = emu.BvhEmu(mesh, nodes, leaf)  # keeps the arrays
    desc = H._lib.SceneDesc()
    desc.points, desc.num_points = mesh.points.ctypes.data, len(mesh.points)
    desc.triangles, desc.num_triangles = mesh.triangles.ctypes.data, len(mesh.triangles)
    desc.materials, desc.num_materials = mesh.materials.ctypes.data, len(mesh.materials)
    desc.nodes, desc.num_nodes = nodes.ctypes.data, len(nodes)
    desc.leaf_data, desc.num_leaf_data = leaf.ctypes.data, len(leaf)
    h = lib.bvhemu_create(C.byref(desc))
    o, d = np.ascontiguousarray(o, np.float32), np.ascontiguousarray(d, np.float32)
    w = np.zeros(5)
    lib.bvhemu_work(h, len(o), o.ctypes.data, d.ctypes.data, w.ctypes.data)
    lib.bvhemu_destroy(h)
    del e
    return w


def _on_the_ground(size, n=100):
    """A sphere of radius 1 over a ground quad of that half width."""
    a, b = np.linspace(0, 2 * np.pi, n, endpoint=False), np.linspace(0, np.pi, n // 2 + 1)
    p = np.array([[np.sin(y) * np.cos(x), np.cos(y) + 1.2, np.sin(y) * np.sin(x)] for y in b for x in a])
    i = (np.arange(n // 2)[:, None] * n + np.arange(n)).ravel()
    j = (np.arange(n // 2)[:, None] * n + (np.arange(n) + 1) % n).ravel()
    t = np.concatenate([np.stack([i, j, i + n], 1), np.stack([j, j + n, i + n], 1)])
    g = size * np.array([[-1, 0, -1], [1, 0, -1], [1, 0, 1], [-1, 0, 1]])
    k = len(p)
    return p, t, _mesh(np.concatenate([p, g]), np.concatenate([t, [[k, k + 1, k + 2], [k, k + 2, k + 3]]]))


@pytest.mark.parametrize("size", [1, 100, 10000, 30000])
def test_small_triangles_in_a_large_scene(size):
    p, t, mesh = _on_the_ground(size)
    rng = np.random.default_rng(1)
    o = np.array([0, 1.2, 0]) + rng.normal(size=(5000, 3)) * 2.5
    d = p[t[rng.integers(0, len(t), 5000)]].mean(1) - o + rng.normal(size=(5000, 3)) * 0.1
    nodes, tests, steps, leaves, walk_tests = _work(mesh, *H.build_kdtree(mesh.points, mesh.triangles), o, d)
    assert nodes < steps and tests < walk_tests / 2, (nodes, tests, steps, leaves, walk_tests)


@pytest.mark.parametrize("name", ["spheres", "terrain", "soup"])
def test_ordinary_rays(name):
    mesh, nodes, leaf = _scene(name)
    for o, d in (S.aabb_random_rays(mesh, 5000, 3), _from_afar(mesh, 5000, 4, 2)):
        visits, tests, steps, leaves, walk_tests = _work(mesh, nodes, leaf, o, d)
        assert visits < steps + leaves and tests < walk_tests, (visits, tests, steps, leaves, walk_tests)
