"""Tile lists on grids of every number of region passes, against the oracle's stable sort of (tile, depth) keys."""
import numpy as np
import pytest
import torch

from radiance_meshes_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,passes", [(128, 256, 1), (136, 256, 2), (2048, 4096, 2), (2200, 3840, 3)])
def test_lists(oracle, cuda_lib, H, W, passes):
    from radiance_meshes_b200 import raster
    from radiance_meshes_b200.render import tcam_to_device
    tcam = scenes.make_tcam(scenes.look_at((0.2, 0.1, 2.6)), H, W, 60.0, tile=2, min_t=0.1)
    regions = -(-tcam["grid_height"] // 4) * -(-tcam["grid_width"] // 8)
    assert passes == (1 if regions <= 256 else 2 if regions <= 65_536 else 3)  # digits of up to 8 bits
    pts = scenes.points_gaussians(3_000, seed=11)
    tets = scenes.delaunay(pts)
    pr = oracle.project(tets, pts, tcam)
    ref_idx, ref_ranges = oracle.build_lists(pr["tiles_touched"], pr["rect"], pr["vs_tetra"], tcam["grid_height"],
                                             tcam["grid_width"])
    dev = torch.device("cuda:0")
    ctx = raster.project_and_bin(torch.tensor(tets, device=dev, dtype=torch.int32), torch.tensor(pts, device=dev),
                                 tcam_to_device(tcam, dev))
    n_keys, _ = raster.read_info(ctx)
    np.testing.assert_array_equal(raster.build_tile_lists(ctx, n_keys).cpu().numpy(), ref_idx)
    np.testing.assert_array_equal(ctx["tile_ranges"].cpu().numpy(), ref_ranges)
