"""The chain rule from record gradients to vertices and cell values, for ranges of tets: a lane per tet up to a million tets,
lists beyond; ranges that begin off the 16-byte grid of the cell-value gradients, as those of a job on several GPUs may."""
import numpy as np
import pytest
import torch

from radiance_meshes_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,begin", [(1, 0), (31, 0), (65, 2), (4_099, 1), (1_000_000, 0), (1_000_001, 0), (1_000_130, 4),
                                     (1_000_900, 313)])
@pytest.mark.parametrize("share", [0.3, 1.0])
def test_range_of_tets(cuda_lib, T, begin, share):
    from radiance_meshes_b200 import _lib, raster
    from radiance_meshes_b200.render import tcam_to_device
    dev, V = torch.device("cuda:0"), 5_000
    gen = torch.Generator(dev).manual_seed(T + begin)
    v = torch.rand((V, 3), generator=gen, device=dev) * 2.0 - 1.0
    idx = torch.randint(0, V, (T, 4), generator=gen, device=dev, dtype=torch.int32)
    a, b, c, d = v[idx.long()].unbind(1)
    flat = (torch.linalg.cross(b - a, c - a) * (d - a)).sum(1).abs() < 1e-3  # which side is outside must not hang on rounding
    v[:4] = torch.tensor([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], device=dev, dtype=torch.float32)
    idx[flat | (idx < 4).any(1)] = torch.tensor([0, 1, 2, 3], device=dev, dtype=torch.int32)
    cell = torch.randn((T, 7), generator=gen, device=dev)
    rows = torch.randn((T, 24), generator=gen, device=dev)
    rows[torch.rand((T,), generator=gen, device=dev) < 0.1] = 0.0  # flagged, but nothing came of it
    flags = (torch.rand((T,), generator=gen, device=dev) < share).to(torch.uint8)
    rows[flags == 0] = float("nan")  # neither cleared nor written
    tcam = scenes.make_tcam(scenes.look_at((0.2, 0.4, 2.5)), 32, 32, 60.0)
    cam = raster.CameraArgs(tcam_to_device(tcam, dev), dev)
    got_v, got_c = torch.zeros((V, 3), device=dev), torch.full((T, 7), -7.0, device=dev)
    none = torch.empty((1,), dtype=torch.int32, device=dev)
    _lib.check(_lib.load().rm_backward_finish(
        *[raster._ptr(t) for t in (idx, v, cell)], begin, T, T, cam.ref, raster._ptr(rows),
        raster.hit_list_ref((none, none, none, flags)), raster._ptr(got_v), raster._ptr(got_c), raster._stream(dev)))

    # the records in 64 bits, differentiated by torch
    v64, c64 = v.double().requires_grad_(True), cell.double().requires_grad_(True)
    eye = torch.tensor(tcam["cam_pos"], device=dev).double()
    on = torch.nonzero(flags[begin:])[:, 0] + begin
    p, q = v64[idx[on].long()], c64[on]
    fields = []
    for i, (base, e1, e2, other) in enumerate([(0, 1, 2, 3), (0, 1, 3, 2), (0, 2, 3, 1), (1, 2, 3, 0)]):
        n = torch.linalg.cross(p[:, e1] - p[:, base], p[:, e2] - p[:, base])
        n = n * -torch.sign((n * (p[:, other] - p[:, base])).sum(1, keepdim=True)).detach()  # outwards
        fields += [n, -(n * (p[:, base] - eye)).sum(1, keepdim=True)]
    fields += [q[:, 4:7], (q[:, 4:7] * (eye - p[:, 0])).sum(1, keepdim=True), q[:, 1:4], torch.relu(q[:, :1])]
    (torch.cat(fields, 1) * rows[on].double()).sum().backward()

    # a term is off by some 32-bit roundings of values of its own size, a vertex sums up to some hundred terms
    assert float((got_v - v64.grad).norm()) <= 1e-5 * float(v64.grad.norm())
    assert bool((got_c[:begin] == -7.0).all())
    torch.testing.assert_close(got_c[begin:], c64.grad[begin:].float(), rtol=1e-5, atol=1e-5)
    assert not got_c[begin:][flags[begin:] == 0].any()
