"""Tile populations from the corners of the rectangles: corners inside and outside the window of a warp's neighbours."""
import numpy as np
import pytest
import torch

from radiance_meshes_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    pts = scenes.points_gaussians(3_000, seed=3)
    return pts, scenes.delaunay(pts)


@pytest.mark.parametrize("order", ["neighbours", "shuffled"])
@pytest.mark.parametrize("H,W,tile,fov", [(64, 60, 4, 60.0),    # 16 x 15 tiles: every corner but the last row in reach
                                          (72, 76, 4, 60.0),    # just outside
                                          (611, 409, 4, 30.0),  # rectangles wider than a window
                                          (200, 333, 2, 60.0), (90, 70, 16, 100.0)])
@pytest.mark.parametrize("n_tets", [1, 31, 33, 129, 10_007])
def test_tile_ranges(cuda_lib, mesh, order, H, W, tile, fov, n_tets):
    from radiance_meshes_b200 import raster
    from radiance_meshes_b200.render import tcam_to_device
    pts, tets = mesh
    if order == "shuffled":
        tets = tets[np.random.default_rng(1).permutation(len(tets))]
    tets = tets[:n_tets]
    tcam = scenes.make_tcam(scenes.look_at((0.2, 0.1, 2.2)), H, W, fov, tile=tile, min_t=0.1)
    dev = torch.device("cuda:0")
    ctx = raster.project_and_bin(torch.tensor(tets, device=dev, dtype=torch.int32), torch.tensor(pts, device=dev),
                                 tcam_to_device(tcam, dev))
    n_keys, n_visible = raster.read_info(ctx)
    rect, touched = ctx["rect"].cpu().numpy(), ctx["tiles_touched"].cpu().numpy()
    count = np.zeros((tcam["grid_height"], tcam["grid_width"]), np.int64)
    for x0, y0, x1, y1 in rect[touched > 0]:
        count[y0:y1, x0:x1] += 1
    count = count.reshape(-1)
    end = np.cumsum(count)
    want = np.where(count[:, None] > 0, np.stack([end - count, end], 1), 0)
    assert n_keys == end[-1] and n_visible == (touched > 0).sum()
    np.testing.assert_array_equal(ctx["tile_ranges"].cpu().numpy(), want)
