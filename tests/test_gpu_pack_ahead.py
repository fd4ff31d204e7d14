"""Records packed while the host waits for the number of list entries, against those packed behind the list build."""
import numpy as np
import pytest
import scene_util
import torch

pytestmark = pytest.mark.gpu


def _inputs(**change):
    pts, tets, cell = scene_util.small_scene(300, seed=6)
    dev = torch.device("cuda:0")
    from radiance_meshes_b200.render import tcam_to_device
    s = dict(indices=torch.tensor(tets, device=dev, dtype=torch.int32), vertices=torch.tensor(pts, device=dev),
             cell=torch.tensor(cell, device=dev), tcam=tcam_to_device(scene_util.camera(H=53, W=61), dev),
             jitter=torch.tensor(scene_util.jitter(53, 61, 2), device=dev))
    s.update({k: f(s[k]) for k, f in change.items()})
    return s


def _frame(s, ahead, grad=True):
    from radiance_meshes_b200.render import render
    v, c = s["vertices"].detach(), s["cell"].detach()
    if grad:
        v, c = v.requires_grad_(True), c.requires_grad_(True)
    pkg = render(s["indices"], v, c, s["tcam"], s["jitter"], before_blend=None if ahead else lambda: None)
    if grad:
        (pkg["image"].sum() + pkg["distortion_img"].sum() + pkg["distortion_loss"]).backward()
    return pkg, v.grad, c.grad


@pytest.mark.parametrize("change", [{}, {"cell": lambda t: t.double()}, {"cell": lambda t: t.t().contiguous().t()},
                                    {"indices": lambda t: t.long()}, {"vertices": lambda t: t.double()},
                                    {"indices": lambda t: t[:1]}, {"tcam": lambda c: dict(c, tile_rows=None)}])
@pytest.mark.parametrize("grad", [True, False])
def test_same_frame(cuda_lib, change, grad):
    """Types, orders and sizes that the blend takes: the same bits, and gradients that differ by the order of their sums (the
    atomics of some hundred tets a vertex: 1e-5)."""
    if "indices" in change:
        change = dict(change, cell=change.get("cell", lambda t: t))
    s = _inputs(**change)
    s["cell"] = s["cell"][:s["indices"].shape[0]]
    (a, va, ca), (b, vb, cb) = _frame(s, True, grad), _frame(s, False, grad)
    for k in ("image", "distortion_img", "sorted_tetra_idx", "tile_ranges", "mask"):
        assert torch.equal(a[k], b[k]), k
    if grad:
        assert float((va - vb).norm()) <= 1e-5 * float(vb.norm()) and float((ca - cb).norm()) <= 1e-5 * float(cb.norm())


@pytest.mark.parametrize("change,error", [({"cell": lambda t: t[:, :4].contiguous()}, AssertionError),
                                          ({"vertices": lambda t: t * float("nan")}, AssertionError),
                                          ({"indices": lambda t: t + 10_000}, IndexError)])
def test_what_was_refused_stays_refused(cuda_lib, change, error):
    s = _inputs(**change)
    for ahead in (True, False):
        with pytest.raises(error):
            _frame(s, ahead, grad=False)
    torch.cuda.synchronize()
    good, _, _ = _frame(_inputs(), True, grad=False)  # a frame given up leaves nothing behind
    assert np.isfinite(good["image"].cpu().numpy()).all()
