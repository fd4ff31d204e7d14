"""Which pair of a hit a plane's gradient is summed from: the entering one for planes that face the camera, the leaving one for the
others, both where the near plane lies behind the camera."""
import pytest

import scene_util
from radiance_meshes_b200 import scenes
from test_gpu_parity import check_against_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [64, 452])  # two lanes per pixel; one, above two waves of half-warps (113 x 113 tiles)
@pytest.mark.parametrize("min_t", [-0.25, 0.0, 0.3])
def test_gradients_with_the_camera_inside_tets(oracle, cuda_lib, min_t, size):
    """The camera is inside the mesh, so that one tet holds it, tets straddle a ray's origin and, with a negative min_t, rays
    enter and leave tets through planes that lie on the same side of the camera.  Tolerances: those of the other gradients."""
    pts, tets, cell = scene_util.small_scene(400, seed=8, zero_frac=0.2)
    tcam = scenes.make_tcam(scenes.look_at((0.05, 0.02, -0.1), (0.4, 0.1, 1.0)), size, size, 90.0, tile=4, min_t=min_t)
    check_against_oracle(oracle, pts, tets, cell, tcam, scene_util.jitter(size, size, 4))
