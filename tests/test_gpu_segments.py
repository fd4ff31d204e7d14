"""Length and weights of a ray's segment in one tet."""
import numpy as np
import pytest
import torch

from radiance_meshes_b200 import scenes

pytestmark = pytest.mark.gpu


def _render(pts, cell, min_t, jitter, size=8):
    """image, distortion moments and the leaves of one tet before a camera at the origin that looks along z."""
    from radiance_meshes_b200.render import render, tcam_to_device
    tcam = tcam_to_device(scenes.make_tcam(np.eye(4), size, size, 40.0, min_t=min_t), "cuda:0")
    v = torch.tensor(pts, dtype=torch.float32, device="cuda:0", requires_grad=True)
    c = torch.tensor(cell, dtype=torch.float32, device="cuda:0")[None].requires_grad_(True)
    pkg = render(torch.tensor([[0, 1, 2, 3]], dtype=torch.int32, device="cuda:0"), v, c, tcam,
                 torch.full((size, size, 2), jitter, device="cuda:0"))
    return pkg["image"], pkg["distortion_img"], v, c


@pytest.mark.parametrize("min_t", [0.1, 0.2, 0.01, 4.05])
@pytest.mark.parametrize("exit_z", [4.25, 6.3125, 8.5, 12.0])
def test_length_is_the_difference_of_the_distances_from_the_origin(cuda_lib, exit_z, min_t):
    """The two distances are rounded where they are shifted from the camera to the ray's origin, and their difference decides
    at which tet a ray ends: the same operations in every build.  The ray along z enters this tet at 4 and leaves it at exit_z;
    both come out of the slab test without rounding (normals, offsets and reciprocals are exact)."""
    pts = [[-2, -2, 4], [6, -2, 4], [-2, 6, 4], [0, 2, 2 * exit_z - 4]]
    image, dist, _, _ = _render(pts, [1.0, 0.5, 0.5, 0.5, 0, 0, 0], min_t, 0.0)
    f = np.float32
    enter, leave = max(f(4) - f(min_t), f(0)), f(exit_z) - f(min_t)
    px = image[4, 4], dist[4, 4]  # its sample is the principal point
    assert px[0][3].item() == -float(leave - enter)
    assert px[1][3].item() == float(f(0.5) * (leave + enter))  # first moment of a density of 1
