"""Negative ids in a caller's tile lists name no tet: the walks pass over them, as if the list were without them."""
import pytest
import torch

from test_gpu_same_bits import _tcam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tets,size,sized", [(600, 97, True), (1500, 97, True),   # two lanes per pixel; lines past L1
                                               (200, 900, True), (200, 900, False)])  # long lists first; two units per warp
def test_negative_ids_are_passed_over(cuda_lib, n_tets, size, sized):
    from radiance_meshes_b200 import _lib, raster
    gen = torch.Generator("cuda").manual_seed(n_tets + size)
    v = 4.0 * torch.rand((400, 3), generator=gen, device="cuda:0") - 2.0
    idx = torch.randint(0, 400, (n_tets, 4), generator=gen, device="cuda:0", dtype=torch.int32)
    cell = torch.rand((n_tets, 7), generator=gen, device="cuda:0") * torch.tensor([0.2, 1, 1, 1, 1, 1, 1], device="cuda:0")
    tcam = _tcam(size, size, 4)
    ctx = raster.project_and_bin(idx, v, tcam)
    n_keys, _ = raster.read_info(ctx)
    lists = raster.build_tile_lists(ctx, n_keys)
    rec = raster.pack_records(idx, v, cell, ctx["cam"], ctx["tiles_touched"])
    none = torch.tensor([-1, -2, -(1 << 31)], device="cuda:0", dtype=torch.int32).repeat(n_keys // 3 + 1)[:n_keys]
    holed = torch.stack([none, lists], 1).reshape(-1)  # one in front of every entry
    per, jitter = torch.rand((2, size, size), generator=gen, device="cuda:0"), torch.rand((size, size, 2), generator=gen, device="cuda:0")

    def walks(ids, ranges):
        def empty(k):
            return torch.empty((size, size, k), device="cuda:0")
        p = raster._ptr
        lib, n, st, cam = _lib.load(), ids.shape[0] if sized else -1, raster._stream(v.device), ctx["cam"].ref
        out, const = [empty(4), empty(5), empty(1).int()], [empty(4), empty(4), empty(1).int()]
        _lib.check(lib.rm_forward_sized(p(ids), p(ranges), p(rec), cam, p(jitter), *[p(t) for t in out], None, n, st))
        _lib.check(lib.rm_forward_constant_color_sized(p(ids), p(ranges), p(rec), cam, 1.5, -0.1, *[p(t) for t in const], n, st))
        stats = raster.tet_err(ids, ranges, rec, ctx["cam"], per[0], per[1], n_tets)
        img, dist, contrib, hits = raster.forward(ids, ranges, rec, ctx["cam"], jitter)
        grads = raster.backward(ids, ranges, rec, ctx["cam"], jitter, img, dist, contrib, hits, torch.ones_like(img),
                                0.01 * torch.ones_like(dist), idx, v, cell)
        return out[:2] + const[:2] + [img, dist, stats[1]], [stats[0], *grads]
    want, want_sums = walks(lists, ctx["tile_ranges"])
    got, got_sums = walks(holed, 2 * ctx["tile_ranges"])
    assert int((want[0][..., 3] < -1.0).sum()) > size
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    # sums of up to 50,000 atomic additions in any order: 2^-24 times the root of their number is 1.3e-5
    for a, b in zip(got_sums, want_sums):
        assert float((a - b).norm()) <= 1e-4 * float(b.norm())
