"""A jitter that has to be converted is the frame's own: what the caller does with it afterwards does not reach the backward
pass."""
import numpy as np
import pytest
import scene_util
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["float64", "permuted", "float16"])
def test_converted_jitter_may_be_refilled_before_the_backward_pass(cuda_lib, form):
    from radiance_meshes_b200.render import render, tcam_to_device
    pts, tets, cell = scene_util.small_scene(300, seed=4)
    dev, H, W = torch.device("cuda:0"), 37, 53
    tcam = tcam_to_device(scene_util.camera(H=H, W=W), dev)
    base = torch.tensor(np.round(scene_util.jitter(H, W, 5) * 256) / 256, device=dev)  # the same in every type
    jit = {"float64": base.double(), "float16": base.half(), "permuted": base.permute(2, 0, 1).contiguous().permute(1, 2, 0)}[form]
    out = []
    for j, refill in ((base, False), (jit, True)):
        v, c = torch.tensor(pts, device=dev, requires_grad=True), torch.tensor(cell, device=dev, requires_grad=True)
        pkg = render(torch.tensor(tets, device=dev), v, c, tcam, j)
        if refill:
            j.fill_(0.25)
        pkg["image"].square().sum().backward()
        out.append((pkg["image"].detach(), v.grad, c.grad))
    assert torch.equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1:], out[1][1:]):  # float atomics: order varies
        assert float((a - b).norm() / b.norm()) < 1e-5
