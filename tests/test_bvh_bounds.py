"""CPU test of the rays for which the hierarchy's boxes have to be larger than
its triangles: the triangle test's rounding accepts rays that pass beside a
triangle, and the answer is still the tree walk's bit for bit."""
import numpy as np
import pytest

import hptracing_b200 as H
from tests import scenes as S
from tests.test_bvh import _check, _mesh, _scene, emu


def _turn(mesh):
    """The mesh turned, so that no plane of it is along an axis."""
    q, _ = np.linalg.qr(np.random.default_rng(1).normal(size=(3, 3)))
    m = _mesh((mesh.points[:, :3] - 0.5) @ q.T, mesh.triangles[:, :3])
    return (m, *H.build_kdtree(m.points, m.triangles))


def _plane(n=40):
    """A tessellated unit square."""
    g = np.stack(np.meshgrid(*2 * [np.linspace(0, 1, n + 1)], indexing="ij"), -1).reshape(-1, 2)
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).ravel()
    return _mesh(np.concatenate([g, np.full((len(g), 1), 0.5)], 1),
                 np.concatenate([np.stack([i, i + 1, i + n + 2], 1), np.stack([i, i + n + 2, i + n + 1], 1)]))


def _corners(mesh, k):
    p = mesh.points[:, :3].astype(np.float64)
    return [p[mesh.triangles[k, j]] for j in range(3)]


def _unit(v):
    return v / np.maximum(np.linalg.norm(v, axis=1, keepdims=True), 1e-30)


def _in_plane(mesh, n, seed):
    """Rays through two points of a triangle's plane: the origin up to a scene
    size away, the other point within three edges."""
    rng = np.random.default_rng(seed)
    a, b, c = _corners(mesh, rng.integers(0, len(mesh.triangles), n))
    p = mesh.points[:, :3].astype(np.float64)
    u = _unit(b - a)
    w = _unit((c - a) - ((c - a) * u).sum(1, keepdims=True) * u)
    away = np.linalg.norm(p.max(0) - p.min(0)) * 10.0 ** rng.uniform(-3, 0, (n, 1))
    x = rng.uniform(-1, 1, (2, n, 1)) * away
    y = rng.uniform(-3, 3, (2, n, 1)) * np.linalg.norm(b - a, axis=1, keepdims=True)
    o = (a + b + c) / 3 + x[0] * u + x[1] * w
    return o, _unit((a + b + c) / 3 + y[0] * u + y[1] * w - o)


def _from_afar(mesh, n, seed, sizes):
    """Rays from that many scene sizes away towards points of triangles."""
    rng = np.random.default_rng(seed)
    tri = _corners(mesh, rng.integers(0, len(mesh.triangles), n))
    q = sum(w[:, None] * v for w, v in zip(rng.dirichlet([1, 1, 1], n).T, tri))
    p = mesh.points[:, :3].astype(np.float64)
    o = (0.5 * (p.min(0) + p.max(0)) + _unit(rng.normal(size=(n, 3))) * sizes * (p.max(0) - p.min(0)).max())
    o = o.astype(np.float32)
    return o, _unit(q - o)


def _along_surface(mesh, n, seed):
    """From a point of a triangle towards another of the same one, as a light
    that samples itself."""
    rng = np.random.default_rng(seed)
    tri = _corners(mesh, rng.integers(0, len(mesh.triangles), n))
    o, q = (sum(w[:, None] * v for w, v in zip(rng.dirichlet([1, 1, 1], n).T, tri)).astype(np.float32)
            for _ in range(2))
    d = _unit((q - o).astype(np.float64)).astype(np.float32)
    return o + np.float32(1e-5) * d, d


@pytest.mark.parametrize("name", ["room", "turned room", "plane", "turned plane", "soup", "degenerate", "spheres",
                                  "terrain"])
def test_rays_in_a_triangles_plane(name):
    scene = {"turned room": lambda: _turn(_scene("room")[0]), "turned plane": lambda: _turn(_plane()),
             "plane": lambda: (lambda m: (m, *H.build_kdtree(m.points, m.triangles)))(_plane())}
    mesh, nodes, leaf = scene.get(name, lambda: _scene(name))()
    e = emu.BvhEmu(mesh, nodes, leaf)
    _check(e.query(*_in_plane(mesh, 40000, 5)))
    _check(e.query(*_along_surface(mesh, 30000, 6)))


@pytest.mark.parametrize("name", ["terrain", "spheres", "room", "degenerate"])
def test_origins_far_away(name):
    """The roundings of boxes, test and certificate grow with the distance."""
    mesh, nodes, leaf = _scene(name)
    e = emu.BvhEmu(mesh, nodes, leaf)
    for sizes in (1.5, 3, 4.2, 10, 100, 1000, 4000, 10000):
        _check(e.query(*_from_afar(mesh, 10000, 7, sizes)))
    # Most rays from a few sizes away do not need the tree.
    assert e.query(*_from_afar(mesh, 4000, 8, 1.5))["certain"].mean() > 0.98


def test_hit_before_its_leaf():
    """In a triangle's plane the computed t may lie before every leaf that has
    the triangle; in the first of them another one may be nearer still."""
    g = _plane(60)
    q, _ = np.linalg.qr(np.random.default_rng(1).normal(size=(3, 3)))
    m = _mesh((g.points[:, :3] - np.float32([0, 0, 0.5])) @ q.T, g.triangles[:, :3])
    e = emu.BvhEmu(m, *H.build_kdtree(m.points, m.triangles))
    o = [[0.05844295769929886, 0.13787004351615906, 0.07542713731527328],
         [-2.018704652786255, 0.4258774518966675, -0.19801566004753113],
         [-1.3616396188735962, -1.131714105606079, -0.7919849753379822],
         [1.0416405200958252, 0.9955244064331055, 0.6660779118537903],
         [0.4593617916107178, 0.31658682227134705, 0.23692654073238373]]
    d = [[-0.5454838275909424, -0.7143399715423584, -0.43836721777915955],
         [0.8948383927345276, 0.31137898564338684, 0.3198552131652832],
         [0.34956181049346924, 0.8218493461608887, 0.4498557448387146],
         [-0.7876143455505371, -0.48537158966064453, -0.3795762062072754],
         [-0.7643405795097351, -0.5145841836929321, -0.3885699212551117]]
    _check(e.query(np.float32(o), np.float32(d)))


def _other_tree(nodes, leaf, count, drop, add, seed):
    """The leaf lists with a share of the entries dropped and some triangles
    added, most of which the leaf does not touch; some entries twice."""
    rng = np.random.default_rng(seed)
    lists, at, used = [], {}, 0
    for off in nodes["data"][(nodes["child"] < 0) & (nodes["data"] >= 0)]:
        ids = leaf[off + 1:off + 1 + leaf[off]]
        ids = ids[rng.random(len(ids)) >= drop]
        more = rng.integers(0, count, rng.binomial(4, add))
        twice = ids[:1] if rng.random() < add else ids[:0]
        ids = np.concatenate([ids, more, twice])
        at[int(off)] = used
        lists.append(np.concatenate([[len(ids)], ids]))
        used += 1 + len(ids)
    nodes = nodes.copy()
    has = (nodes["child"] < 0) & (nodes["data"] >= 0)
    nodes["data"][has] = [at[int(x)] for x in nodes["data"][has]]
    return nodes, np.concatenate(lists).astype(np.int32)


@pytest.mark.parametrize("name", ["nine", "soup", "room", "flat"])
@pytest.mark.parametrize("drop,add", [(0.1, 0), (0.5, 0), (0.9, 0), (0, 0.5), (0.3, 0.2)])
def test_tree_with_other_lists(name, drop, add):
    """A caller's tree need not list a triangle in the leaves it touches, and
    may list it in others: the answer is that tree's."""
    mesh, nodes, leaf = _scene(name)
    nodes, leaf = _other_tree(nodes, leaf, len(mesh.triangles), drop, add, 3)
    e = emu.BvhEmu(mesh, nodes, leaf)
    _check(e.query(*S.aabb_random_rays(mesh, 20000, 3)))
    _check(e.query(*_in_plane(mesh, 5000, 4)))


@pytest.mark.parametrize("name", ["soup", "degenerate", "room", "turned room", "spheres", "flat"])
def test_directions_along_edges(name):
    """Along a triangle's edge e2 the test divides zero by zero, and where
    nothing else is hit the tree walk answers t = +inf."""
    mesh, nodes, leaf = _turn(_scene("room")[0]) if name == "turned room" else _scene(name)
    e = emu.BvhEmu(mesh, nodes, leaf)
    rng = np.random.default_rng(8)
    p = mesh.points[:, :3]
    k = rng.integers(0, len(mesh.triangles), 20000)
    along = (p[mesh.triangles[k, 2]] - p[mesh.triangles[k, 0]]).astype(np.float32)
    o = rng.uniform(p.min(0), p.max(0), (20000, 3)).astype(np.float32)
    for d in (along, along * np.float32(0.5), -along, _unit(along.astype(np.float64))):
        _check(e.query(o, d))


def test_axis_rays_that_miss_do_not_need_the_tree():
    mesh, nodes, leaf = _scene("soup")
    e = emu.BvhEmu(mesh, nodes, leaf)
    rng = np.random.default_rng(3)
    p = mesh.points[:, :3]
    q = e.query(rng.uniform(p.min(0), p.max(0), (5000, 3)), np.eye(3)[rng.integers(0, 3, 5000)])
    _check(q)
    assert q["certain"][q["tri"] < 0].mean() > 0.99


@pytest.mark.parametrize("name", ["far", "soup", "spheres", "terrain", "room", "flat"])
def test_rays_almost_along_a_split_plane(name):
    """The tree walk finds its leaves by rounded points: within rounding of a
    split plane it may go along its other side, where the filter rejects."""
    mesh, nodes, leaf = _scene(name)
    rng = np.random.default_rng(0)
    n, p = 60000, mesh.points[:, :3]
    faces = np.concatenate([nodes["box_start"].reshape(len(nodes), -1)[:, :3],
                            nodes["box_end"].reshape(len(nodes), -1)[:, :3]]).astype(np.float32)
    axis = rng.integers(0, 3, n)
    x, ulps = faces[rng.integers(0, len(faces), n), axis], rng.integers(-3, 4, n)
    for k in range(3):
        to = np.where(ulps > k, np.inf, np.where(ulps < -k, -np.inf, x)).astype(np.float32)
        x = np.nextafter(x, to)
    grow = 0.2 * (p.max(0) - p.min(0))
    o = rng.uniform(p.min(0) - grow, p.max(0) + grow, (n, 3)).astype(np.float32)
    o[np.arange(n), axis] = x
    d = rng.normal(size=(n, 3))
    d[np.arange(n), axis] *= 10.0 ** rng.uniform(-8, -1, n)
    _check(emu.BvhEmu(mesh, nodes, leaf).query(o, _unit(d)))


@pytest.mark.parametrize("scale", [1e-14, 1e-12, 1e-8, 1e8, 1e12])
@pytest.mark.parametrize("length", [1e-14, 1e-8, 1e8, 1e14])
def test_scenes_and_directions_of_extreme_size(scale, length):
    """Where products of the test leave the normal numbers, its error is not
    relative any more."""
    g = _scene("nine")[0] if scale * length > 1e24 else S.make_scene(3, seed=2, family=2, target_triangles=2000)[0]
    m = _mesh(g.points[:, :3].astype(np.float64) * scale, g.triangles[:, :3])
    e = emu.BvhEmu(m, *H.build_kdtree(m.points, m.triangles))
    for o, d in (_in_plane(m, 20000, 5), S.aabb_random_rays(m, 10000, 3)):
        _check(e.query(o, d * np.float32(length)))
