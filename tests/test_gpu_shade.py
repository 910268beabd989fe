"""GPU tests of the shading pass over several jobs: the counts a warp keeps for
one job, and one scene for all jobs against a scene per job."""
import numpy as np
import pytest

import hptracing_b200 as H
from tests import scenes as S

pytestmark = pytest.mark.gpu


def _params(n, spp, seed):
    return H.make_params(n, 3, 1, 1, (0.1, 0.2, 0), spp, 5, 0, 1.0, seed)


@pytest.mark.parametrize("sizes", [[1], [31, 1, 33], [8] * 40, [257, 5, 1024, 2]])
@pytest.mark.parametrize("scenes", [1, 2])
def test_jobs_of_a_batch_shade_alike(built, sizes, scenes):
    """Warps that hold one job's paths, several jobs' or a change from one to
    the next: every job as rendered alone, bit for bit, and the same number of
    rays traced."""
    if H.device_count() == 0:
        pytest.skip("no CUDA device")
    gpus = [H.Scene(*S.make_scene(0)), H.Scene(*S.make_scene(0))][:scenes]
    cam = S.hp_camera(S.ROOM_CAM)
    alone, rays = [], 0
    for k, n in enumerate(sizes):
        b = H.Batch()
        b.add(gpus[0], cam, _params(n, 1 + k % 3, k), want_accum=True)
        alone.append(b.run()[0][1])
        rays += b.stats()["intersect_queries"]
    batch = H.Batch()
    for k, n in enumerate(sizes):
        batch.add(gpus[k % scenes], cam, _params(n, 1 + k % 3, k), want_accum=True)
    out = batch.run()
    assert batch.stats()["intersect_queries"] == rays
    for a, o in zip(alone, out):
        assert np.array_equal(a, o[1])
