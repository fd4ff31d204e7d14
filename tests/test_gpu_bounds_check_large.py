"""The bounds-checked build on frames and meshes that take the kernels of the larger sizes: walks by halves and with the long
lists first, the backward walk by halves, the sorts with 16 items per thread and ordinary launches, three region passes."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import sys
    import numpy as np
    import torch
    sys.path.insert(0, {root!r})
    from radiance_meshes_b200 import _lib, raster, scenes
    from radiance_meshes_b200.render import render, tcam_to_device
    from delaunay_rasterization.internal.alphablend_tiled_slang import AlphaBlendTiledRender as ConstantColour
    from delaunay_rasterization.internal.render_err import tet_error_stats
    from delaunay_rasterization.internal.render_grid import RenderGrid
    assert _lib.bounds_checked(), "the bounds-checked build was not loaded"
    dev, wave = torch.device("cuda:0"), 5920

    def mesh(points):
        pts = scenes.points_gaussians(points, seed=points)
        tets = scenes.delaunay(pts)
        return pts, tets, scenes._features(np.random.default_rng(points), tets.shape[0], 2.0, 1.5, 0.3)

    def frame(m, H, W, tile):
        pts, tets, cell = m
        tcam = tcam_to_device(scenes.make_tcam(scenes.look_at((0.0, 0.3, 3.2)), H, W, 50.0, tile=tile, min_t=0.1), dev)
        v, c = torch.tensor(pts, device=dev, requires_grad=True), torch.tensor(cell, device=dev, requires_grad=True)
        idx = torch.tensor(tets, device=dev, dtype=torch.int32)
        pkg = render(idx, v, c, tcam, torch.rand((H, W, 2), device=dev))
        (pkg["image"].sum() + 0.1 * pkg["distortion_img"].sum()).backward()
        lists, ranges = pkg["sorted_tetra_idx"], pkg["tile_ranges"]
        tet_error_stats(lists, ranges, idx, v.detach(), c.detach(), tcam, torch.rand((H, W), device=dev),
                        torch.rand((H, W), device=dev), pkg["mask"].to(torch.int32))
        grid = RenderGrid(H, W, tile_height=tile, tile_width=tile)
        rgbs = c.detach()[:, [1, 2, 3, 0]].contiguous().requires_grad_(True)
        img, dist = ConstantColour.apply(lists, ranges, idx, v, rgbs, grid, tcam, 100, -0.1)
        (img.sum() + dist.sum()).backward()
        torch.cuda.synchronize()
        lens = (ranges[:, 1] - ranges[:, 0]).float()
        ctx = raster.project_and_bin(idx, v, tcam)
        raster.read_info(ctx)
        return (ranges.shape[0] * ((tile * tile + 15) // 16), float(lens.mean()), float(lens.max()), tets.shape[0],
                ctx["n_region_keys"])

    small, large = mesh(300), mesh(24_000)
    units, mean, longest, _, _ = frame(small, 560, 563, 4)
    assert 2 * wave < units <= 8 * wave and mean < 64, "by halves"
    units, mean, longest, _, _ = frame(small, 900, 901, 4)
    assert units > 8 * wave and longest > 3 * mean, "long lists first"
    units, mean, longest, _, _ = frame(small, 603, 1206, 5)
    assert units > 8 * wave and longest > 3 * mean, "long lists first, two units per tile"
    _, _, _, tets, pairs = frame(large, 540, 720, 4)
    assert min(tets, pairs) > 131_072, "16 items per thread, ordinary launches"
    # more than 65,536 regions of 8 x 4 tiles
    pts, tets, _ = mesh(1_000)
    tcam = tcam_to_device(scenes.make_tcam(scenes.look_at((0.2, 0.1, 2.6)), 2200, 3840, 60.0, tile=2, min_t=0.1), dev)
    ctx = raster.project_and_bin(torch.tensor(tets, device=dev, dtype=torch.int32), torch.tensor(pts, device=dev), tcam)
    n_keys, _ = raster.read_info(ctx)
    raster.build_tile_lists(ctx, n_keys)
    print("STATUS", _lib.bounds_status())
""")


def test_bounds_checked_build_stays_clean_on_large_frames(cuda_lib):
    from radiance_meshes_b200.csrc import build
    env = dict(os.environ, RM_B200_LIBRARY=build.build(variant="check"))
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    status = int(out.stdout.split("STATUS")[1])
    assert status == 0, f"bounds violations, site bits {status:#x}"
