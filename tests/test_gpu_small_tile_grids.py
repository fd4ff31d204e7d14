"""Tile grids so small that the tile coverage is collected in several partial arrays: 1 to 512 of them."""
import numpy as np
import pytest
import torch

from radiance_meshes_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    pts = scenes.points_gaussians(21_000, seed=5)
    return pts, scenes.delaunay(pts)


@pytest.mark.parametrize("H,W,tile", [(7, 9, 16), (33, 16, 16), (203, 130, 16)])
@pytest.mark.parametrize("n_tets", [1, 511, 512, 13_000, 131_072])  # one array, two from 512 tets on, many
def test_lists(oracle, cuda_lib, mesh, H, W, tile, n_tets):
    from radiance_meshes_b200 import raster
    from radiance_meshes_b200.render import tcam_to_device
    pts, tets = mesh[0], mesh[1][:n_tets]
    tcam = scenes.make_tcam(scenes.look_at((0.2, 0.1, 2.6)), H, W, 60.0, tile=tile, min_t=0.1)
    pr = oracle.project(tets, pts, tcam)
    ref_idx, ref_ranges = oracle.build_lists(pr["tiles_touched"], pr["rect"], pr["vs_tetra"], tcam["grid_height"],
                                             tcam["grid_width"])
    dev = torch.device("cuda:0")
    ctx = raster.project_and_bin(torch.tensor(tets, device=dev, dtype=torch.int32), torch.tensor(pts, device=dev),
                                 tcam_to_device(tcam, dev))
    n_keys, _ = raster.read_info(ctx)
    np.testing.assert_array_equal(raster.build_tile_lists(ctx, n_keys).cpu().numpy(), ref_idx)
    np.testing.assert_array_equal(ctx["tile_ranges"].cpu().numpy(), ref_ranges)
