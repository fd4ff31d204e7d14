"""Tile lists so long that their hull lines are copied past L1: the same bits as through it."""
import pytest
import torch

from test_gpu_same_bits import _forward, _tcam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tets,size,long", [(1500, 97, True), (1500, 900, True),  # two lanes per pixel; long lists first
                                              (600, 97, False)])                     # the other side of the line
def test_same_bits(cuda_lib, n_tets, size, long):
    """Large tets in any order, most of which cover most of the view.  A call that does not say how long its lists are copies
    through L1."""
    gen = torch.Generator("cuda").manual_seed(n_tets + size)
    v = 4.0 * torch.rand((400, 3), generator=gen, device="cuda:0") - 2.0
    idx = torch.randint(0, 400, (n_tets, 4), generator=gen, device="cuda:0", dtype=torch.int32)
    cell = torch.rand((n_tets, 7), generator=gen, device="cuda:0") * torch.tensor([0.02, 1, 1, 1, 1, 1, 1], device="cuda:0")
    cell[::7, 0] = 0.0
    tcam = _tcam(size, size, 4)
    jitter = torch.rand((size, size, 2), generator=gen, device="cuda:0")
    sized, n_keys = _forward((idx, v, cell), tcam, jitter)
    assert (n_keys >= 800 * tcam["grid_width"] * tcam["grid_height"]) == long
    unsized, _ = _forward((idx, v, cell), tcam, jitter, sized=False)
    assert int((sized[2] > 300).sum()) > size  # entries walked
    for a, b in zip(sized, unsized):
        assert torch.equal(a, b)
