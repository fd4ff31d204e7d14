"""Waits of the sorts that run out: in the checked build a block waits for no look-back word and never sees those of every
other block; it counts what is missing itself, as the ordinary build does after some milliseconds.  The lists have to be
the oracle's all the same."""
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
    from oracle import oracle
    from radiance_meshes_b200 import _lib, raster, scenes
    from radiance_meshes_b200.render import tcam_to_device
    assert _lib.bounds_checked(), "the checked build was not loaded"
    dev = torch.device("cuda:0")
    pts = scenes.points_gaussians(21_000, seed=5)
    all_tets = scenes.delaunay(pts)
    seen = 0
    # 4 and 16 items per thread, one region pass and two, launches behind one another and ordinary ones
    for n_tets, H, W, tile in [(1025, 203, 317, 4), (65_536, 203, 317, 4), (131_073, 203, 317, 4), (131_073, 1080, 1920, 4)]:
        tets = all_tets[:n_tets]
        tcam = scenes.make_tcam(scenes.look_at((0.2, 0.1, 2.6)), H, W, 60.0, tile=tile, min_t=0.1)
        pr = oracle.project(tets, pts, tcam)
        ref_idx, ref_ranges = oracle.build_lists(pr["tiles_touched"], pr["rect"], pr["vs_tetra"], tcam["grid_height"],
                                                 tcam["grid_width"])
        ctx = raster.project_and_bin(torch.tensor(tets, device=dev, dtype=torch.int32), torch.tensor(pts, device=dev),
                                     tcam_to_device(tcam, dev))
        n_keys, _ = raster.read_info(ctx)
        lists = raster.build_tile_lists(ctx, n_keys)
        np.testing.assert_array_equal(lists.cpu().numpy(), ref_idx)
        np.testing.assert_array_equal(ctx["tile_ranges"].cpu().numpy(), ref_ranges)
        seen |= _lib.load().rm_debug_recounted()
    print("RECOUNTED", seen, _lib.bounds_status())
""")


def test_lists_are_right_when_no_wait_is_long_enough(cuda_lib, oracle):
    from radiance_meshes_b200.csrc import build
    env = dict(os.environ, RM_B200_LIBRARY=build.build(variant="check"))
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    seen, status = [int(x) for x in out.stdout.split("RECOUNTED")[1].split()]
    assert seen == 15, "a kind of wait never ran out, so that its count was not tested"
    assert status == 0
