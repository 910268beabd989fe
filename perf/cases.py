"""Timed workloads of the path tracer, one pass each through the public API.

A case is a dict of plain values. `prepare` gives what a renderer's host has
in hand before the call (a device-resident scene, a camera pose, a batch or
a server, host or device arrays), `run` is one call sequence as such a host
makes it, `work` the bytes and operations it cannot do without.

The scene families and cameras are those of hptracing_b200.scenes. The mesh
and the tree of a scene are generated once per process (they stand for a
loaded file). A scene below 500k triangles is put on the device by every
`prepare`, the 2.4M-triangle terrain once per process, as a viewer or a
server keeps it resident. The seed moves the camera and keys the random
streams, so frames of different seeds trace different paths.
"""
import ctypes
import math

import numpy as np
import torch

import hptracing_b200 as H
from hptracing_b200 import scenes as S

RESIDENT_TRIANGLES = 500_000
# Triangles of the nominal scenes ("scaled" scenes name their own count).
TRIANGLES = {"room": 36, "spheres": 61_476, "terrain": 2_413_060}


def listed():
    return [
        # The smallest useful call: a thumbnail or first preview of a scene
        # being set up. Launches and host latency count.
        dict(name="room_thumb", kind="render", scene="room", w=64, h=48, spp=1, depth=5, accum=False),
        # The box-room frame: a scene of a few dozen triangles (the classic
        # Cornell-like set-up) at an ordinary preview size.
        dict(name="room_frame", kind="render", scene="room", w=256, h=256, spp=16, depth=5, accum=True),
        # A pose request of an interactive viewer: one camera move at 4 spp.
        dict(name="spheres_pose", kind="render", scene="spheres", w=512, h=512, spp=4, depth=6, accum=False),
        # The ordinary frame: 61k textured triangles, 64 spp, depth 8.
        dict(name="spheres_frame", kind="render", scene="spheres", w=512, h=512, spp=64, depth=8, accum=True),
        # An equirectangular panorama from inside the scene.
        dict(name="spheres_pano", kind="render", scene="spheres", w=1024, h=512, spp=16, depth=6,
             accum=False, pano=True),
        # Odd sizes, supersampling, another tessellation, direct light only.
        dict(name="odd_supersampled", kind="render", scene="scaled", family=1, triangles=20_011, w=333, h=217,
             ss=2, spp=7, depth=5, accum=True, no_diffuse=True),
        # A full-HD frame of a 2.4M-triangle landscape that stays resident.
        dict(name="terrain_frame", kind="render", scene="terrain", w=1920, h=1080, spp=4, depth=8, accum=False),
        # Many small jobs over several scenes in one wavefront (a dataset of
        # renders: sizes, samples and depths vary from job to job).
        dict(name="batch_mixed", kind="batch", jobs=24, top=256, spp_top=16, depth_top=10),
        # A server with two resident scenes: a burst of pose requests and
        # two panoramas, pumped until every image is out.
        dict(name="serve_mixed", kind="serve", poses=16, pose=512, spp=4, panos=2, pano_h=384, pano_spp=8, depth=6),
        # Closest hits of incoherent rays for a host that runs its own loop.
        dict(name="intersect_spheres", kind="intersect", scene="spheres", n=1_048_579),
        # Shading and next direction of a batch of hits, host arrays.
        dict(name="shade_spheres", kind="shade", scene="spheres", n=262_147),
        # Stable compaction of a device flag array, half of it set.
        dict(name="compact_device", kind="compact", n=33_554_432, density=0.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scene(rng, large=True):
    x = rng.random()
    if x < 0.2:
        return dict(scene="room")
    if x < 0.5:
        return dict(scene="spheres")
    if x < 0.58 and large:
        return dict(scene="terrain")
    return dict(scene="scaled", family=rng.choice([1, 1, 2]), triangles=_log_int(rng, 2_000, 400_000))


def draw(rng):
    x = rng.random()
    if x < 0.06:
        return dict(kind="compact", n=_log_int(rng, 1_000, 33_554_432), density=round(rng.uniform(0.02, 0.98), 3))
    if x < 0.13:
        return dict(kind="shade", n=_log_int(rng, 1_000, 400_000), **_draw_scene(rng, large=False))
    if x < 0.23:
        return dict(kind="intersect", n=_log_int(rng, 1_000, 1_048_579), **_draw_scene(rng, large=False))
    if x < 0.31:
        return dict(kind="batch", jobs=rng.randint(3, 24), top=_log_int(rng, 48, 256), spp_top=rng.choice([1, 4, 16]),
                    depth_top=rng.randint(3, 10))
    if x < 0.39:
        return dict(kind="serve", poses=rng.randint(1, 16), pose=_log_int(rng, 64, 512), spp=rng.randint(1, 4),
                    panos=rng.randint(0, 2), pano_h=_log_int(rng, 64, 384), pano_spp=rng.randint(1, 8),
                    depth=rng.randint(3, 6))
    while True:
        c = dict(kind="render", w=_log_int(rng, 48, 1920), h=_log_int(rng, 48, 1080), spp=_log_int(rng, 1, 64),
                 depth=rng.randint(3, 10), accum=rng.random() < 0.5, **_draw_scene(rng))
        if rng.random() < 0.2:
            c["ss"] = 2
        if rng.random() < 0.15:
            c["no_diffuse"] = True
        if c["scene"] in ("room", "spheres") and rng.random() < 0.2:
            c.update(pano=True, w=2 * c["h"])
        # Path segments, weighted by what a large scene's cost more: at most
        # those of the full-HD terrain frame.
        big = c["scene"] == "terrain" or c.get("triangles", 0) > 100_000
        cost = c["w"] * c["h"] * c.get("ss", 1) ** 2 * c["spp"] * c["depth"] * (2 if big else 1)
        if cost <= 1920 * 1080 * 4 * 8 * 2:
            return c


# --- scenes -----------------------------------------------------------------

_meshes = {}
_resident = {}


def _key(case):
    return (case["scene"], case.get("family", 0), case.get("triangles", 0))


def _mesh(key):
    """(mesh, tree nodes, leaf list) of a scene, generated once."""
    if key not in _meshes:
        scene, family, triangles = key
        if scene == "scaled":
            _meshes[key] = S.make_scene(3, seed=5, family=family, target_triangles=triangles)
        else:
            _meshes[key] = S.make_scene({"room": 0, "spheres": 1, "terrain": 2}[scene], seed=0)
    return _meshes[key]


def _device_scene(key):
    mesh, nodes, leaf = _mesh(key)
    if len(mesh.triangles) < RESIDENT_TRIANGLES:
        return H.Scene(mesh, nodes, leaf)
    if key not in _resident:
        _resident[key] = H.Scene(mesh, nodes, leaf)
    return _resident[key]


def _camera(key, rng, pano=False, aspect=1.0):
    """The family's camera, moved and turned a little by the seed."""
    scene, family, _ = key
    if pano:
        c = dict(S.PANO_CAM)
        move = 0.05
    elif scene == "terrain" or (scene == "scaled" and family == 2):
        c = dict(S.terrain_cam(aspect))
        move = 0.03
    else:
        c = dict(S.ROOM_CAM)
        c["width"] = c["height"] * aspect
        move = 0.03
    c["view_p"] = tuple(float(v) for v in np.asarray(c["view_p"]) + rng.uniform(-move, move, 3))
    if not pano:
        a = rng.uniform(-0.05, 0.05)
        right, top = np.asarray(c["right_dir"], float), np.asarray(c["top_dir"], float)
        c["right_dir"] = tuple(float(v) for v in math.cos(a) * right + math.sin(a) * np.cross(top, right))
    return S.hp_camera(c)


def _params(w, h, ss, spp, depth, seed, key, no_diffuse=False):
    bg = (0.2, 0.2, 0.2) if key[0] == "terrain" or key[1] == 2 else (0.0, 0.0, 0.0)
    return H.make_params(w, h, ss, ss, bg, spp, depth, int(no_diffuse), 1.0, seed)


# --- prepare ----------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind == "render":
        key = _key(case)
        pano = case.get("pano", False)
        return dict(kind=kind, scene=_device_scene(key), accum=case["accum"],
                    camera=_camera(key, rng, pano, case["w"] / case["h"]),
                    params=_params(case["w"], case["h"], case.get("ss", 1), case["spp"], case["depth"], seed, key,
                                   case.get("no_diffuse", False)))
    if kind == "batch":
        keys = [("room", 0, 0), ("spheres", 0, 0), ("scaled", 2, 100_000)]
        scenes = [_device_scene(k) for k in keys]
        jobs = []
        for j in range(case["jobs"]):
            k = int(rng.integers(len(keys)))
            res = max(32, case["top"] >> int(rng.integers(0, 3)))
            spp = max(1, case["spp_top"] >> int(rng.integers(0, 3)))
            depth = int(rng.integers(min(3, case["depth_top"]), case["depth_top"] + 1))
            jobs.append((scenes[k], _camera(keys[k], rng), _params(res, res, 1, spp, depth, seed + j, keys[k])))
        return dict(kind=kind, batch=H.Batch(0), jobs=jobs)
    if kind == "serve":
        keys = [("room", 0, 0), ("spheres", 0, 0)]
        server = H.Server(0, max_jobs=32, memory_budget=1 << 30, capacity=1 << 20, large_inflight_pct=25)
        slots = [server.add_scene(_device_scene(k)) for k in keys]
        reqs = []
        for j in range(case["poses"] + case["panos"]):
            k = j % 2
            if j < case["poses"]:
                reqs.append((slots[k], _camera(keys[k], rng), _params(case["pose"], case["pose"], 1, case["spp"],
                                                                      case["depth"], seed + j, keys[k])))
            else:
                reqs.append((slots[k], _camera(keys[k], rng, pano=True),
                             _params(2 * case["pano_h"], case["pano_h"], 1, case["pano_spp"], case["depth"],
                                     seed + j, keys[k])))
        return dict(kind=kind, server=server, reqs=reqs)
    if kind == "intersect":
        key = _key(case)
        origins, directions = _rays(key, case["n"], rng)
        return dict(kind=kind, scene=_device_scene(key), origins=origins, directions=directions)
    if kind == "shade":
        key = _key(case)
        return dict(kind=kind, scene=_device_scene(key), **_hits(key, case["n"], rng))
    n = case["n"]
    flags = torch.from_numpy((rng.random(n, dtype=np.float32) < case["density"]).astype(np.int32)).cuda()
    return dict(kind="compact", flags=flags, out=torch.zeros(n, dtype=torch.int32, device="cuda"),
                count=torch.zeros(1, dtype=torch.int32, device="cuda"))


def _unit(rng, n):
    d = rng.normal(size=(n, 3))
    return (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _rays(key, n, rng):
    """Origins in the scene's bounding box, directions all around."""
    points = _mesh(key)[0].points[:, :3]
    return rng.uniform(points.min(0), points.max(0), (n, 3)).astype(np.float32), _unit(rng, n)


def _hits(key, n, rng):
    """Hits as an intersect stage reports them: points all over the mesh,
    seen from a distance within the scene's size."""
    mesh = _mesh(key)[0]
    points = mesh.points[:, :3].astype(np.float64)
    tris = rng.integers(0, len(mesh.triangles), n).astype(np.int32)
    a, b, c = (points[mesh.triangles[tris, k]] for k in range(3))
    u, v = rng.random((2, n, 1))
    flip = u + v > 1
    u, v = np.where(flip, 1 - u, u), np.where(flip, 1 - v, v)
    d = _unit(rng, n)
    t = rng.uniform(0.05, 1.0, n).astype(np.float32)
    origins = (a + u * (b - a) + v * (c - a) - t[:, None] * d.astype(np.float64)).astype(np.float32)
    return dict(origins=origins, directions=d, strengths=rng.uniform(0.1, 1.0, (n, 3)).astype(np.float32),
                tris=tris, ts=t, seeds=rng.integers(0, 1 << 48, n, dtype=np.uint64))


# --- run --------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "render":
        return state["scene"].render(state["camera"], state["params"], want_accum=state["accum"])
    if kind == "batch":
        batch = state["batch"]
        for scene, camera, params in state["jobs"]:
            batch.add(scene, camera, params, want_accum=True)
        # One array for all images and one for all accumulators.
        done = batch.run()
        return [np.concatenate([rgba.ravel() for rgba, _ in done]), np.concatenate([acc.ravel() for _, acc in done])]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(*r) for r in state["reqs"]]
        while server.pending():
            server.pump(4)
        images = []
        for rid, (_, _, p) in zip(ids, state["reqs"]):
            rgba = np.empty((p.sample_y, p.sample_x, 4), np.uint8)
            server.poll(rid, rgba)
            images.append(rgba.ravel())
        return np.concatenate(images)
    if kind == "intersect":
        return state["scene"].intersect(state["origins"], state["directions"])
    if kind == "shade":
        hit = state["scene"].shade(state["origins"], state["directions"], state["strengths"], state["tris"],
                                   state["ts"], state["seeds"])
        following = state["scene"].next_dir(hit["branch"], state["directions"], hit["hit_p"], hit["normal"],
                                            hit["strength"], hit["param"], hit["seeds"])
        # Seeds are 48-bit: as signed words they are the same numbers.
        for r in (hit, following):
            r["seeds"] = r["seeds"].view(np.int64)
        return [hit, following]
    flags, out, count = state["flags"], state["out"], state["count"]
    H._lib.check(H.lib().hpt_compact_noalloc(
        ctypes.c_void_p(flags.data_ptr()), flags.numel(), ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(count.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return [out, count]


# --- work -------------------------------------------------------------------

def _triangles(case):
    return case.get("triangles") or TRIANGLES[case["scene"]]


def work(case):
    """Bytes: each input (the scene's 64 bytes per triangle among them) read
    once, each output written once. Operations: per path at least one
    segment, with one ray-triangle test (about 60) and its shading (about
    190); the number of bounces is not known beforehand."""
    kind = case["kind"]
    per_segment = 250.0
    if kind == "render":
        pixels = case["w"] * case["h"]
        rays = pixels * case.get("ss", 1) ** 2
        return {"bytes": 64.0 * _triangles(case) + 4 * pixels + (12 * rays if case["accum"] else 0),
                "flops": per_segment * rays * (1 + case["spp"])}
    if kind == "batch":
        rays = case["jobs"] * (case["top"] / 2.0) ** 2
        return {"bytes": 64.0 * 160_000 + 16 * rays, "flops": per_segment * rays * (1 + case["spp_top"] / 2.0)}
    if kind == "serve":
        poses, panos = case["poses"] * case["pose"] ** 2, case["panos"] * 2 * case["pano_h"] ** 2
        return {"bytes": 64.0 * 61_512 + 4 * (poses + panos),
                "flops": per_segment * (poses * (1 + case["spp"]) + panos * (1 + case["pano_spp"]))}
    if kind == "intersect":
        return {"bytes": 64.0 * _triangles(case) + (24 + 16) * case["n"], "flops": 60.0 * case["n"]}
    if kind == "shade":
        return {"bytes": 48.0 * _triangles(case) + (52 + 64 + 60 + 48) * case["n"], "flops": 190.0 * case["n"]}
    return {"bytes": 4.0 * case["n"] * (1 + case["density"]), "flops": 0.0}


# --- exact ------------------------------------------------------------------

def exact(case, seed):
    """Rendered radiance has no 64-bit value: a path's next bounce depends on
    the last bits of the one before it. The closest hits of a few dozen
    triangles and the hit points of the shading stage have one."""
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "shade":
        h = _hits(_key(case), case["n"], rng)
        hit = dict.fromkeys(("contrib", "branch", "normal", "strength", "param", "seeds"))
        hit["hit_p"] = h["origins"].astype(np.float64) + h["ts"].astype(np.float64)[:, None] * h["directions"]
        return [hit, dict.fromkeys(("origins", "directions", "strength", "alive", "seeds"))]
    if case["kind"] == "intersect" and case["scene"] == "room":
        key = _key(case)
        mesh = _mesh(key)[0]
        o, d = (x.astype(np.float64) for x in _rays(key, case["n"], rng))
        best = [np.full(len(o), np.inf), np.zeros(len(o)), np.zeros(len(o))]
        # Edge vectors as the stage keeps them: differences in 32 bits.
        corners = [mesh.points[mesh.triangles[:, k], :3] for k in range(3)]
        for a, e1, e2 in zip(corners[0], corners[1] - corners[0], corners[2] - corners[0]):
            a, e1, e2 = (x.astype(np.float64) for x in (a, e1, e2))
            p = np.cross(d, e2)
            with np.errstate(divide="ignore", invalid="ignore"):
                inv = 1.0 / (p @ e1)
                to = o - a
                u = (to * p).sum(1) * inv
                q = np.cross(to, e1)
                v = (d * q).sum(1) * inv
                t = (q @ e2) * inv
                hit = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (t < best[0])
            for have, new in zip(best, (t, u, v)):
                have[hit] = new[hit]
        best[0][np.isinf(best[0])] = 0.0
        return [None, *best]
    return None
