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


def _exact(pts, cell, min_t, size):
    """image[H,W,3] of the same tet in 64 bits, with its leaves: the closed form of alpha = exp(-x), phi = (1 - alpha)/x,
    colour = (phi - alpha) c(exit) + (1 - phi) c(entry) for a linear colour field c."""
    tcam = scenes.make_tcam(np.eye(4), size, size, 40.0)
    fx, cx = float(tcam["K"][0, 0]), float(tcam["K"][0, 2])
    v = torch.tensor(pts, dtype=torch.float32, device="cuda:0").double().requires_grad_(True)
    c = torch.tensor(cell, dtype=torch.float32, device="cuda:0").double().requires_grad_(True)
    p = (torch.arange(size, dtype=torch.float64, device="cuda:0") + 0.5 - cx) / fx
    d = torch.stack([p[None, :].expand(size, size), p[:, None].expand(size, size), torch.ones(size, size, device="cuda:0").double()], -1)
    d = d / d.norm(dim=-1, keepdim=True)
    enter = torch.full((size, size), float(np.float32(min_t)), dtype=torch.float64, device="cuda:0")
    leave = torch.full_like(enter, 1e30)
    for i in range(4):
        a, b, e = [v[k] for k in range(4) if k != i]
        n = torch.linalg.cross(b - a, e - a)
        n = n * torch.sign(((a - v[i]) * n).sum()).detach()  # outwards
        den = (n * d).sum(-1)
        t = (n * a).sum() / den
        enter = torch.where(den < 0, torch.maximum(enter, t), enter)
        leave = torch.where(den < 0, leave, torch.minimum(leave, t))
    x = c[0] * (leave - enter)
    assert bool((x > 0).all())  # the tet covers the view
    alpha, phi = torch.exp(-x), -torch.expm1(-x) / x
    at = lambda t: c[1:4] + ((t[..., None] * d - v[0]) * c[4:7]).sum(-1, keepdim=True)  # noqa: E731
    return (phi - alpha)[..., None] * at(leave) + (1.0 - phi)[..., None] * at(enter), v, c


# Two lanes per pixel (8 x 8), and more than two waves of units, whose backward pass takes a lane per pixel.  64 pixels of either
# have a gradient, so that the sums stay short.  The distances are known to 3e-7 of themselves, the segment to some 1e-6, and
# the weights go with up to the square of it: 1e-5.
@pytest.mark.parametrize("size", [8, 448])
@pytest.mark.parametrize("depth", [1e-3, 0.1, 0.2, 0.3, 1.0, 10.0, 1e2, 1e3, 1e4, 1e6])
def test_weights_of_thin_and_thick_segments(cuda_lib, depth, size):
    """Image and gradients through one tet of 0.001 to a million optical depths: the weight of the exit falls as 1 / x, the
    gradient of the density as 1 / x^2, and both keep their relative precision."""
    pts = [[-2, -2, 4], [6, -2, 4], [-2, 6, 4], [0.25, 2, 9]]
    cell = [0.5 * depth, 0.3, 0.6, 0.2, 0.4, -0.3, 0.7]
    image, _, v, c = _render(pts, cell, 0.1, 0.5, size)
    exact, ve, ce = _exact(pts, cell, 0.1, size)
    step = size // 8
    image[step // 2::step, step // 2::step, :3].sum().backward()
    exact[step // 2::step, step // 2::step].sum().backward()

    def off(a, b):
        return float((a.double() - b).norm() / b.norm())
    assert off(image[..., :3].detach(), exact.detach()) < 2e-6
    got = dict(density=off(c.grad[0, :1], ce.grad[:1]), colours=off(c.grad[0, 1:], ce.grad[1:]), vertices=off(v.grad, ve.grad))
    assert max(got.values()) < 1e-5, got
