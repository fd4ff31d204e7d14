"""An image has the same bits however its units of 16 pixels are dealt to warps, which depends on the size of the call: a frame
in one call, the same frame in bands of rows, and calls that do not say how long the lists are."""
import numpy as np
import pytest
import torch

from radiance_meshes_b200 import scenes

pytestmark = pytest.mark.gpu
WAVE = 5920  # units that the chip holds at a time


def _scene(points):
    pts = scenes.points_gaussians(points, seed=points)
    tets = scenes.delaunay(pts)
    cell = scenes._features(np.random.default_rng(points), tets.shape[0], 2.0, 1.5, 0.3)
    dev = torch.device("cuda:0")
    return torch.tensor(tets, device=dev, dtype=torch.int32), torch.tensor(pts, device=dev), torch.tensor(cell, device=dev)


def _tcam(H, W, tile, **kw):
    from radiance_meshes_b200.render import tcam_to_device
    return tcam_to_device(scenes.make_tcam(scenes.look_at((0.0, 0.3, 3.2)), H, W, 50.0, tile=tile, min_t=0.1, **kw), "cuda:0")


def _forward(scene, tcam, jitter, rows=None, sized=True):
    """(image, distortion, contributors, list length) of the rows."""
    from radiance_meshes_b200 import _lib, raster
    idx, v, cell = scene
    ctx = raster.project_and_bin(idx, v, tcam, tile_rows=rows)
    n_keys, _ = raster.read_info(ctx)
    lists = raster.build_tile_lists(ctx, n_keys)
    rec = raster.pack_records(idx, v, cell, ctx["cam"], ctx["tiles_touched"])
    H, W = tcam["image_height"], tcam["image_width"]
    out = [torch.zeros((H, W, k), dtype=t, device=v.device) for k, t in ((4, torch.float32), (5, torch.float32), (1, torch.int32))]
    _lib.check(_lib.load().rm_forward_sized(
        *[raster._ptr(t) for t in (lists, ctx["tile_ranges"], rec)], ctx["cam"].ref, raster._ptr(jitter),
        *[raster._ptr(t) for t in out], None, n_keys if sized else -1, raster._stream(v.device)))
    return out, n_keys


@pytest.mark.parametrize("points,H,W,tile,kw", [
    (300, 900, 900, 4, {}),                                            # short lists: bands of 2 to 8 waves go by halves
    (3000, 1600, 1601, 4, {}),                                         # long lists: they go by pairs; ragged right edge
    (3000, 1100, 1200, 5, dict(distortion=[0.06, 0.01, 0.001, -0.0005])),  # two units per tile, the second one ragged; a lens
    (1000, 1300, 1300, 4, dict(camera_type=1))])
def test_frame_and_bands(cuda_lib, points, H, W, tile, kw):
    scene, tcam = _scene(points), _tcam(H, W, tile, **kw)
    jitter = torch.rand((H, W, 2), generator=torch.Generator("cuda").manual_seed(points), device="cuda:0")
    per_row = tcam["grid_width"] * ((tile * tile + 15) // 16)
    rows = tcam["grid_height"]
    assert rows * per_row > 8 * WAVE  # long lists first
    full, _ = _forward(scene, tcam, jitter)
    assert bool((full[0][..., 3] < -5.5).any())  # some pixels end before their list does
    ways = set()
    for band in (2 * WAVE // per_row, 5 * WAVE // per_row):
        for r in range(0, rows, band):
            b = (r, min(r + band, rows))
            part, n_keys = _forward(scene, tcam, jitter, rows=b)
            units, tiles = (b[1] - b[0]) * per_row, (b[1] - b[0]) * tcam["grid_width"]
            ways.add("pairs" if units <= 2 * WAVE or n_keys >= 64 * tiles else "halves")
            y = slice(tile * b[0], min(tile * b[1], H))
            for got, want in zip(part, full):
                assert torch.equal(got[y], want[y]), b
    assert "pairs" in ways
    unsized, _ = _forward(scene, tcam, jitter, sized=False)  # by halves throughout
    for got, want in zip(unsized, full):
        assert torch.equal(got, want)


@pytest.mark.parametrize("H,tile", [(600, 8), (601, 16)])
def test_constant_color(cuda_lib, H, tile):
    """About 4 waves: by pairs if the caller says how long the lists are, else by halves."""
    from radiance_meshes_b200 import _lib, raster
    idx, v, cell = _scene(5000)
    cell[:, 4:] = 0.0
    ctx = raster.project_and_bin(idx, v, _tcam(H, H, tile))
    n_keys, _ = raster.read_info(ctx)
    lists = raster.build_tile_lists(ctx, n_keys)
    assert n_keys >= 64 * ctx["G"] and ctx["G"] * tile * tile / 16 > 2 * WAVE
    rec = raster.pack_records(idx, v, cell, ctx["cam"])
    out = []
    for n_list in (n_keys, -1):
        o = [torch.empty((H, H, k), dtype=t, device="cuda:0") for k, t in ((4, torch.float32), (4, torch.float32), (1, torch.int32))]
        _lib.check(_lib.load().rm_forward_constant_color_sized(
            raster._ptr(lists), raster._ptr(ctx["tile_ranges"]), raster._ptr(rec), ctx["cam"].ref, 1.5, -0.1,
            *[raster._ptr(t) for t in o], n_list, raster._stream(v.device)))
        out.append(o)
    assert bool((out[0][0][..., 3] < 1.0 / 255.0).any())
    for a, b in zip(*out):
        assert torch.equal(a, b)
