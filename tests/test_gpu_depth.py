"""GPU test of deep frames: no more iterations than the paths need."""
import numpy as np
import pytest

import hptracing_b200 as H
from tests import scenes as S

pytestmark = pytest.mark.gpu


def _render(scene, depth, capacity=None):
    if capacity:
        t = scene.tuning()
        t.capacity = capacity
        scene.set_tuning(t)
    out = scene.render(S.hp_camera(S.terrain_cam(4 / 3)),
                       H.make_params(64, 48, 1, 1, (0.1, 0.2, 0), 1, depth, 0, 1.0, 3), want_accum=True)
    return out, scene.stats()


def test_depth_beyond_the_longest_path(built):
    if H.device_count() == 0:
        pytest.skip("no CUDA device")
    scene = H.Scene(*S.make_scene(3, seed=2, family=2, target_triangles=4000))
    (rgba, accum), deep = _render(scene, 255)
    lo, hi = 1, 255  # the smallest depth that cuts off no path
    while lo < hi:
        mid = (lo + hi) // 2
        if _render(scene, mid)[1]["intersect_queries"] == deep["intersect_queries"]:
            hi = mid
        else:
            lo = mid + 1
    assert lo < 200
    # 16 ahead, then two batches of 4 until the flag is seen.
    assert deep["iterations"] <= max(lo, 16) + 12, (lo, deep["iterations"])
    # The same bits where paths are started as others end.
    (rgba2, accum2), _ = _render(scene, 255, capacity=1024)
    assert np.array_equal(rgba, rgba2) and np.array_equal(accum, accum2)
