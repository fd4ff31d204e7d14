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


@pytest.fixture
def packed_ahead(monkeypatch):
    """Of every call of pack_ahead that `render` makes, whether it has packed."""
    from radiance_meshes_b200 import render as module
    calls, pack_ahead = [], module.pack_ahead

    def spy(*args):
        packed = pack_ahead(*args)
        calls.append(packed is not None)
        return packed
    monkeypatch.setattr(module, "pack_ahead", spy)
    return calls


@pytest.mark.parametrize("change", [{}, {"cell": lambda t: t.double()}, {"cell": lambda t: t.t().contiguous().t()},
                                    {"indices": lambda t: t.long()}, {"vertices": lambda t: t.double()},
                                    {"indices": lambda t: t[:1]}, {"tcam": lambda c: dict(c, tile_rows=None)}])
@pytest.mark.parametrize("grad", [True, False])
def test_same_frame(cuda_lib, packed_ahead, change, grad):
    """Types, orders and sizes that the blend takes: the same bits, and gradients that differ by the order of their sums (the
    atomics of some hundred tets a vertex: 1e-5)."""
    s = _inputs(**change)
    s["cell"] = s["cell"][:s["indices"].shape[0]]
    a, va, ca = _frame(s, True, grad)
    assert packed_ahead == [True]
    b, vb, cb = _frame(s, False, grad)
    assert packed_ahead == [True]
    for k in ("image", "distortion_img", "sorted_tetra_idx", "tile_ranges", "mask"):
        assert torch.equal(a[k], b[k]), k
    if grad:
        assert float((va - vb).norm()) <= 1e-5 * float(vb.norm()) and float((ca - cb).norm()) <= 1e-5 * float(cb.norm())


@pytest.mark.parametrize("change,error,packs", [({"cell": lambda t: t[:, :4].contiguous()}, AssertionError, False),
                                                ({"vertices": lambda t: t * float("nan")}, AssertionError, True),
                                                ({"indices": lambda t: t + 10_000}, IndexError, True)])
def test_what_was_refused_stays_refused(cuda_lib, packed_ahead, change, error, packs):
    s = _inputs(**change)
    for ahead in (True, False):
        with pytest.raises(error):
            _frame(s, ahead, grad=False)
    assert packed_ahead == [packs]
    torch.cuda.synchronize()
    good, _, _ = _frame(_inputs(), True, grad=False)  # a frame given up leaves nothing behind
    assert np.isfinite(good["image"].cpu().numpy()).all()


def _many_tets(T):
    """T small tets, among them many copies of the same ones, for a 32 x 32 image."""
    from radiance_meshes_b200.render import tcam_to_device
    gen = torch.Generator("cuda").manual_seed(3)
    v = (4.0 * torch.rand((1024, 1, 3), generator=gen, device="cuda:0") - 2.0 +
         0.02 * torch.rand((1024, 4, 3), generator=gen, device="cuda:0")).reshape(-1, 3).contiguous()
    first = 4 * torch.randint(0, 1024, (T, 1), generator=gen, device="cuda:0")
    return dict(indices=(first + torch.arange(4, device="cuda:0")).to(torch.int32), vertices=v,
                cell=torch.rand((T, 7), generator=gen, device="cuda:0"), tcam=tcam_to_device(scene_util.camera(H=32, W=32), "cuda:0"),
                jitter=torch.tensor(scene_util.jitter(32, 32, 5), device="cuda:0"))


def _peak(call):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = call()
    torch.cuda.synchronize()
    del out
    return torch.cuda.max_memory_allocated() - before


@pytest.mark.parametrize("grad", [False, True])
def test_large_mesh_needs_no_more_memory(cuda_lib, packed_ahead, grad):
    """One tet above the limit: records beside the list scratch would be 46 MB more at the peak of a frame alone."""
    from radiance_meshes_b200 import raster
    s = _many_tets(raster.PACK_AHEAD_TETS + 1)
    _frame(s, True, grad)
    assert packed_ahead == [True] * grad
    assert _peak(lambda: _frame(s, True, grad)) <= _peak(lambda: _frame(s, False, grad)) + 2**20


def test_large_mesh_of_the_constant_colour_renderer_needs_no_more_memory(cuda_lib):
    from delaunay_rasterization.internal.alphablend_tiled_slang import AlphaBlendTiledRender, render_constant_color
    from delaunay_rasterization.internal.render_grid import RenderGrid
    from delaunay_rasterization.internal.tile_shader_slang import vertex_and_tile_shader
    from radiance_meshes_b200 import raster
    s = _many_tets(raster.PACK_AHEAD_TETS + 1)
    rgbs, tcam = s["cell"][:, :4], s["tcam"]

    class camera:
        image_height = image_width = 32
        to_dict = staticmethod(lambda device: {k: tcam[k] for k in (
            "world_view_transform", "K", "cam_pos", "distortion_params", "image_height", "image_width", "fovy", "fovx", "camera_type")})

    def whole():
        return render_constant_color(s["indices"], s["vertices"], None, camera, cell_values=rgbs, tile_size=4)

    def stages():  # records behind the list build
        grid = RenderGrid(32, 32, tile_height=4, tile_width=4)
        ids, ranges, vs, cc, mask, _ = vertex_and_tile_shader(s["indices"], s["vertices"], tcam, grid)
        return vs, cc, mask, AlphaBlendTiledRender.apply(ids, ranges, s["indices"], s["vertices"], rgbs, grid, tcam, 100, -0.1)
    whole(), stages()
    assert _peak(whole) <= _peak(stages) + 2**20
