"""Meshes of more than a million tets, where packing works through lists of the tets that need a record, against the same tets in
a small mesh, where a thread packs every tet.  (The chain rule lists its tets in either; test_gpu_chain_rule.py has it against
64 bits.)"""
import numpy as np
import pytest
import torch

import scene_util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,real", [(1_000_001, "spread"), (1_000_192, "front"), (1_000_703, "back")])
def test_large_mesh_equals_small(cuda_lib, T, real):
    from radiance_meshes_b200 import raster
    from radiance_meshes_b200.render import render, tcam_to_device
    pts, tets, cell = scene_util.small_scene(n_points=400, seed=4)  # a fifth of the tets has no density
    n, H, W = len(tets), 45, 51
    at = {"spread": np.sort(np.random.default_rng(2).permutation(T)[:n]), "front": np.arange(n),
          "back": np.arange(T - n, T)}[real]
    big_tets = np.tile(np.arange(len(pts), len(pts) + 4, dtype=np.int32), (T, 1))  # behind the camera: culled
    pts = np.concatenate([pts, np.array([[0, 0, 90], [1, 0, 90], [0, 1, 90], [0, 0, 91]], np.float32)])
    big_cell = np.ones((T, 7), np.float32)
    big_tets[at], big_cell[at] = tets, cell
    tcam = tcam_to_device(scene_util.camera(H=H, W=W), "cuda:0")
    out = []
    for t, c in ((tets, cell), (big_tets, big_cell)):
        t = torch.tensor(t, device="cuda:0", dtype=torch.int32)
        v = torch.tensor(pts, device="cuda:0", requires_grad=True)
        c = torch.tensor(c, device="cuda:0", requires_grad=True)
        pkg = render(t, v, c, tcam, torch.tensor(scene_util.jitter(H, W), device="cuda:0"))
        ctx = raster.project_and_bin(t, v.detach(), tcam)
        rec = raster.pack_records(t, v.detach(), c.detach(), ctx["cam"], ctx["tiles_touched"])
        (pkg["image"].square().sum() + pkg["distortion_img"].sum()).backward()
        out.append((pkg["image"].detach(), pkg["distortion_img"].detach(), rec.reshape(-1), ctx["tiles_touched"] > 0,
                    v.grad, c.grad))
    small, big = out
    assert torch.equal(small[0], big[0]) and torch.equal(small[1], big[1])
    # tets 2k and 2k + 1 share 288 bytes; of a tet without density only the last sector is written
    at = torch.tensor(at, device="cuda:0")
    assert torch.equal(small[3], big[3][at]) and int(big[3].sum()) == int(small[3].sum())
    visible = torch.nonzero(small[3])[:, 0]
    dense = torch.tensor(cell[:, 0] > 0, device="cuda:0")[visible]

    def rows(records, tet):
        return records[(36 * tet - 4 * (tet & 1))[:, None] + torch.arange(32, device="cuda:0")].view(torch.int32)
    a, b = rows(small[2], visible), rows(big[2], at[visible])
    assert torch.equal(a[dense], b[dense]) and torch.equal(a[~dense][:, 24:], b[~dense][:, 24:]) and int((~dense).sum()) > 50
    # sums of at most a few thousand float atomics in another order
    for g, h in ((small[4], big[4]), (small[5], big[5][at])):
        assert float((g - h).norm()) <= 1e-5 * float(g.norm())
    others = torch.ones(T, dtype=torch.bool, device="cuda:0")
    others[at] = False
    assert not big[5][others].any()
