"""A frame that is given up between its two halves: the page-locked memory that the device is about to write goes back only
when it has been written."""
import pytest
import scene_util
import torch

pytestmark = pytest.mark.gpu


def _begin(stream):
    from radiance_meshes_b200 import raster
    from radiance_meshes_b200.render import tcam_to_device
    pts, tets, _ = scene_util.small_scene(300, seed=4)
    dev = torch.device("cuda:0")
    tcam = tcam_to_device(scene_util.camera(), dev)
    idx, v = torch.tensor(tets, device=dev, dtype=torch.int32), torch.tensor(pts, device=dev)
    with torch.cuda.stream(stream):
        # a frame before the one that is looked at: what the first one of a process loads and allocates may take longer than the sleep
        raster.read_info(raster.project_and_bin(idx, v, tcam, host_info=True))
        torch.cuda._sleep(1)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)  # some 50 ms that the frame waits behind
        return raster.project_and_bin(idx, v, tcam, host_info=True)


def test_dropped_context(cuda_lib):
    stream = torch.cuda.Stream()
    ctx = _begin(stream)
    assert not stream.query()  # the frame has not begun
    del ctx
    assert stream.query()


def test_info_is_that_of_the_frame_whichever_stream_reads_it(cuda_lib):
    from radiance_meshes_b200 import raster
    stream = torch.cuda.Stream()
    ctx = _begin(stream)
    n_keys, n_visible = raster.read_info(ctx)  # on the default stream, which has nothing to wait for
    assert stream.query()
    assert raster.read_info(ctx) == (n_keys, n_visible) and n_visible == int(ctx["visible"].sum()) > 0
    assert n_keys == int(ctx["tiles_touched"].sum())
