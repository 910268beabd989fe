"""GPU test of rays of zero strength, which may be answered without a look at
the tree only where every answer adds zero to their path."""
import numpy as np
import pytest

import hptracing_b200 as H
from tests import scenes as S

pytestmark = pytest.mark.gpu


def _with_infinite_material(mesh):
    """The same scene with one more material, of infinite emission, that no
    triangle has: then no ray is answered by its strength."""
    m = np.concatenate([mesh.materials, mesh.materials[:1]])
    m["emission"][-1] = np.inf
    return H.Mesh(mesh.points, mesh.triangles, m, normals=mesh.normals, texcoords=mesh.texcoords,
                  lights=mesh.lights, texture_data=mesh.texture_data, texture_dims=mesh.texture_dims)


@pytest.mark.parametrize("background", [(0.1, 0.2, 0.0), (np.inf, 0.1, np.nan)])
def test_zero_strength_rays_answer_as_all_others(built, background):
    if H.device_count() == 0:
        pytest.skip("no CUDA device")
    mesh, nodes, leaf = S.make_scene(0)
    out = []
    for m in (mesh, _with_infinite_material(mesh)):
        scene = H.Scene(m, nodes, leaf)
        out.append(scene.render(S.hp_camera(S.ROOM_CAM), H.make_params(160, 120, 1, 1, background, 8, 6, 0, 1.0, 5),
                                want_accum=True))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1], equal_nan=True)
