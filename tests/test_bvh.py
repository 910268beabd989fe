"""CPU test of the closest-hit query through the wide hierarchy (bvh.cuh,
bvh_build.cpp): the tree walk's answer bit for bit, over the ray sets and the
trees where it could go wrong."""
import numpy as np
import pytest

import hptracing_b200 as H
import oracle as O
from tests import scenes as S

emu = pytest.importorskip("tests.bvhemu")


def _mesh(points, triangles):
    mat = np.zeros(1, H.MATERIAL_DTYPE)
    tri = np.concatenate([np.asarray(triangles, np.int32), np.zeros((len(triangles), 1), np.int32)], 1)
    return H.Mesh(np.asarray(points, np.float32), tri, mat)


def _soup(n, seed, size=0.1, flat=False):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1, (n, 1, 3))
    p = c + rng.uniform(-size, size, (n, 3, 3))
    if flat:  # axis-aligned triangles in a few shared planes
        ax = rng.integers(0, 3, n)
        p[np.arange(n), :, ax] = (rng.integers(0, 4, n) / 4.0)[:, None]
    return _mesh(p.reshape(-1, 3), np.arange(3 * n).reshape(n, 3))


def _scene(name):
    if name == "room":
        return S.make_scene(0)
    if name == "spheres":
        return S.make_scene(1, seed=1, texture_size=16)
    if name == "terrain":
        return S.make_scene(3, seed=2, family=2, target_triangles=30000)
    mesh = {"one": lambda: _soup(1, 1), "two": lambda: _soup(2, 2), "nine": lambda: _soup(9, 3),
            "soup": lambda: _soup(3000, 4), "flat": lambda: _soup(600, 5, flat=True),
            # Every triangle twice: each hit is a tie.
            "double": lambda: _mesh(np.tile(_soup(200, 6).points[:, :3], (2, 1)), np.arange(1200).reshape(-1, 3)),
            # Far from the origin: coordinates 1e4 times the triangles.
            "far": lambda: _mesh(_soup(500, 7).points[:, :3] + np.float32(1000), np.arange(1500).reshape(-1, 3)),
            # Slivers and zero-area triangles among ordinary ones.
            "degenerate": lambda: _mesh(
                np.where(np.arange(900)[:, None] % 9 == 2, np.roll(_soup(300, 8).points[:, :3], 1, 0),
                         _soup(300, 8).points[:, :3]) * np.float32([1, 1, 0.01]), np.arange(900).reshape(-1, 3)),
            }[name]()
    return (mesh, *H.build_kdtree(mesh.points, mesh.triangles))


def _rays(mesh, nodes):
    cam = [O.raygen(S.ROOM_CAM, 64, 64, 1, 1), O.raygen(S.PANO_CAM, 48, 24, 1, 1),
           S.aabb_random_rays(mesh, 6000, 3)]
    cam += [r for r in S.edge_rays(mesh, nodes, n=400).values()]
    # Directions with components down to denormals.
    rng = np.random.default_rng(9)
    o, d = S.aabb_random_rays(mesh, 500, 4)
    d[np.arange(500), rng.integers(0, 3, 500)] *= (10.0 ** rng.uniform(-42, -6, 500)).astype(np.float32)
    cam.append((o, d))
    cam.append((o, d * np.float32(1e-3)))
    return [np.concatenate(x) for x in zip(*cam)]


def _check(q):
    assert q["flags"] == 0
    bad = (q["tri"] != q["walk_tri"]) | (q["t"].view(np.int32) != q["walk_t"].view(np.int32))
    assert not bad.any(), (np.flatnonzero(bad)[:5], q["tri"][bad][:5], q["walk_tri"][bad][:5])


@pytest.mark.parametrize("name", ["one", "two", "nine", "room", "soup", "flat", "double", "far", "degenerate",
                                  "spheres", "terrain"])
def test_query_is_the_tree_walks(name):
    mesh, nodes, leaf = _scene(name)
    e = emu.BvhEmu(mesh, nodes, leaf)
    assert e.shape()["depth"] < 31
    q = e.query(*_rays(mesh, nodes))
    _check(q)
    if name in ("spheres", "terrain", "soup"):
        # Most rays do not need the tree.
        o, d = S.aabb_random_rays(mesh, 4000, 5)
        assert e.query(o, d)["certain"].mean() > 0.98


def test_tree_that_lists_fewer_triangles():
    """A caller's tree need not list a triangle in every leaf it touches: the
    answer is still that tree's (here every third leaf drops one entry)."""
    mesh, nodes, leaf = _scene("soup")
    leaf = leaf.copy()
    for k, off in enumerate(nodes["data"][(nodes["child"] < 0) & (nodes["data"] >= 0)]):
        count = leaf[off]
        if k % 3 == 0 and count > 1:
            leaf[off + count] = leaf[off + 1]  # the last entry gives way to a repeat of the first
    e = emu.BvhEmu(mesh, nodes, leaf)
    _check(e.query(*_rays(mesh, nodes)))
