"""Host side of the rasterizer: torch tensors in, C-ABI calls, torch tensors out.

PyTorch is used for device memory, streams and autograd plumbing only; every
computation happens in the CUDA library, and the calls of a frame are made by the
compiled host path (csrc/rm_torch.cpp).
"""
import ctypes as C

import torch

from . import _lib


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _stream(device):
    return C.c_void_p(torch.cuda.current_stream(device).cuda_stream)


class CameraArgs:
    """RmCamera plus the device tensors it points at (kept alive with it)."""

    def __init__(self, tcam, device, tile_rows=None):
        self.native = _lib.native().Camera(tcam, device, tile_rows)
        self.address = self.native.address
        self.band_rows_only = self.native.band_rows_only
        self._c = None

    @property
    def c(self):
        if self._c is None:
            self._c = _lib.RmCamera.from_address(self.address)
        return self._c

    @property
    def ref(self):
        return C.byref(self.c)


def _require_cuda(t, name):
    if not (isinstance(t, torch.Tensor) and t.is_cuda):
        raise RuntimeError(f"{name} must be a CUDA tensor (the rasterizer has no CPU path)")


def project_and_bin(indices, vertices, tcam, tile_rows=None, host_info=False):
    """Stage 1 and tile populations. Returns a dict of outputs plus the binning context.  With `host_info` the counters
    also arrive in page-locked memory, where read_info(ctx) finds them without a copy."""
    _require_cuda(indices, "indices")
    _require_cuda(vertices, "vertices")
    cam = CameraArgs(tcam, vertices.device, tile_rows)
    out, pending = _lib.native().project_and_bin(indices, vertices, cam.address, host_info)
    indices, verts, tiles_touched, rect, vs_tetra, circumcenter, tile_ranges, info, ws, visible = out
    gh, gw = cam.native.grid
    return dict(indices=indices, vertices=verts, cam=cam, tiles_touched=tiles_touched, rect=rect, vs_tetra=vs_tetra,
                circumcenter=circumcenter, tile_ranges=tile_ranges, info=info, workspace=ws, visible=visible,
                host_info=pending, T=indices.shape[0], V=verts.shape[0], G=gh * gw)


def read_info(ctx):
    """The one host synchronisation of the binning stage: N, visible count, status."""
    if ctx.get("host_info") is not None:
        n_keys, ctx["n_region_keys"], n_visible, status = ctx["host_info"].wait()
    else:
        n_keys, ctx["n_region_keys"], second = ctx["info"].tolist()
        n_visible = second & 0xFFFFFFFF
        status = (second >> 32) & 0xFFFFFFFF
    if status & _lib.RM_STATUS_NAN_VERTEX:
        # same message as the reference's assert (tile_shader_slang.py:78)
        raise AssertionError("Tensor contains NaN values!")
    if status & _lib.RM_STATUS_BAD_INDEX:
        raise IndexError("rm_b200: indices name a vertex outside [0, n_vertices)")
    if status & _lib.RM_STATUS_KEY_OVERFLOW or n_keys > 2**31 - 1:
        raise RuntimeError(f"rm_b200: {n_keys} (tile, tet) pairs exceed the int32 range of the tile lists")
    return n_keys, n_visible


def build_tile_lists(ctx, n_keys):
    if n_keys > 0 and "n_region_keys" not in ctx:
        raise RuntimeError("rm_b200: call read_info(ctx) before build_tile_lists")
    return _lib.native().build_tile_lists(ctx["rect"], ctx["tile_ranges"], ctx["workspace"], ctx["cam"].address, n_keys,
                                          ctx.get("n_region_keys", 0))


# Up to this many tets the records are packed before the tile lists are built, while the host waits for their length.  They are
# then alive beside the list scratch (peak of a frame without a backward pass, MB, packed ahead and behind: 1M tets 294 and 240,
# 2M 900 and 734, 6.7M 2408 and 1920, 36M 13570 and 10720), for the same 7 to 15 us at every size: 60k tets 170.6 us for 180.1,
# 0.6M 642 for 652, 1M 605 for 612; but 2M 2249 for 2257, 6.7M 2774 for 2788, 36M 14.83 ms for 14.85, within what runs differ by.
PACK_AHEAD_TETS = 1_000_000


def packs_ahead(indices, *differentiable):
    """Whether to pack ahead.  A frame whose backward pass follows does at any size: its peak is that pass's either way (6.7M tets
    3416 MB, 21M 8677; 4.64 ms for 4.66 and 8.64 for 8.68)."""
    return indices.shape[0] <= PACK_AHEAD_TETS or (torch.is_grad_enabled() and any(t.requires_grad for t in differentiable))


def pack_records(indices, vertices, cell_values, cam, tiles_touched=None):
    return _lib.native().pack_records(indices, vertices, cell_values, cam.address, tiles_touched, None, None)


def hit_list_ref(hits):
    """ctypes argument for a hit list given as the (counts, ids, masks) tensors forward() returns."""
    if hits is None:
        return None
    counts, ids, masks, tet_flags = hits
    return C.byref(_lib.RmHitList(_ptr(counts), _ptr(ids), _ptr(masks), _ptr(tet_flags)))


def forward(sorted_idx, tile_ranges, records, cam, ray_jitter, want_hit_masks=True):
    """Returns (output_img, distortion_img, n_contributors, hits); hits = (counts int32 [G*S], ids int32 [N*S],
    masks int16 [N*S + 16*G*S], tet_flags uint8 [T]) are the hit lists backward() walks, None if not requested."""
    flags = None
    if want_hit_masks:
        flags = torch.zeros((max(int(records.shape[0]), 1),), dtype=torch.uint8, device=records.device)
    out = _lib.native().forward(sorted_idx, tile_ranges, records, cam.address, cam.native.zero_fill, ray_jitter, flags)
    return out[0], out[1], out[2], (tuple(out[3:]) + (flags,)) if want_hit_masks else None


# Optional consumer of finished gradients, set by a multi-GPU job (dist.OverlappedGradientSum.install): the
# backward pass then finishes the tets in `chunks` ranges and hands every finished range of cell_values_grad,
# and vertices_grad at the end, to `sink` while the next range is still being finished.
_gradient_sink = None


def set_gradient_sink(sink, chunks=4):
    """sink(tensor) is called on the backward pass's stream, in order, with views of the two gradients as
    they become final: ranges of rows of the cell-value gradients first, the vertex gradients last;
    sink.done() once at the end.  Both gradients live in one buffer (vertex gradients first, zero-padded to a
    multiple of 4 floats, then the cell-value gradients), so the views are contiguous ranges of it.  Optional methods: sink.allocate(n_floats, device) -> a float32 tensor the gradients are
    written to (or None for an ordinary allocation), sink.export(flat) -> the tensor handed to the caller
    after done().  None removes the sink."""
    global _gradient_sink
    _gradient_sink = None if sink is None else (sink, max(1, int(chunks)))


def backward(sorted_idx, tile_ranges, records, cam, ray_jitter, output_img, distortion_img, n_contributors,
             hits, grad_output_img, grad_distortion_img, indices, vertices, cell_values):
    if _gradient_sink is None:
        return _lib.native().backward(sorted_idx, tile_ranges, records, cam.address, ray_jitter, output_img, distortion_img,
                                      n_contributors, *hits, grad_output_img, grad_distortion_img, indices, vertices,
                                      cell_values)
    lib = _lib.load()
    dev = records.device
    T, V = indices.shape[0], vertices.shape[0]
    grad_output_img, grad_distortion_img = grad_output_img.contiguous(), grad_distortion_img.contiguous()
    with torch.cuda.device(dev):
        grad_records = torch.empty((T, _lib.RM_GRAD_RECORD_FLOATS), dtype=torch.float32, device=dev)
        # both gradients live in one allocation (the second one 16-byte aligned), so that a multi-GPU
        # job can sum them over the ranks with a single all-reduce (dist.allreduce_gradients)
        off = (3 * V + 3) // 4 * 4
        sink = _gradient_sink
        flat = None
        if hasattr(sink[0], "allocate"):  # a sink may want the gradients in memory of its own
            flat = sink[0].allocate(off + 7 * T, dev)
        if flat is None:
            flat = torch.empty((off + 7 * T,), dtype=torch.float32, device=dev)
        vertices_grad = flat[:3 * V].view(V, 3)
        cell_grad = flat[off:].view(T, 7)
        if off > 3 * V:
            flat[3 * V:off].zero_()
        href = hit_list_ref(hits)
        st = _stream(dev)
        if _lib.bounds_checked():
            _lib.set_extents(list=sorted_idx.shape[0], tets=T, verts=V, hit_ids=hits[1].shape[0],
                             hit_masks=hits[2].shape[0], units=hits[0].shape[0])
        _lib.check(lib.rm_backward_integrate(_ptr(tile_ranges), _ptr(records), cam.ref, _ptr(ray_jitter),
                                             _ptr(output_img), _ptr(distortion_img), href, _ptr(grad_output_img),
                                             _ptr(grad_distortion_img), T, V, _ptr(grad_records), _ptr(vertices_grad),
                                             st))
        n_chunks = sink[1] if T >= 4096 else 1
        step = -(-T // n_chunks)
        step = -(-step // 256) * 256  # range starts on multiples of 256 tets
        t0 = 0
        while True:
            t1 = min(t0 + step, T)
            _lib.check(lib.rm_backward_finish(_ptr(indices), _ptr(vertices), _ptr(cell_values), t0, t1, T, cam.ref,
                                              _ptr(grad_records), href, _ptr(vertices_grad), _ptr(cell_grad), st))
            if t1 > t0:
                sink[0](cell_grad[t0:t1])
            t0 = t1
            if t0 >= T:
                break
        sink[0](vertices_grad)
        sink[0].done()
        if hasattr(sink[0], "export"):  # the sums leave the sink's memory before its next use
            flat = sink[0].export(flat)
            vertices_grad = flat[:3 * V].view(V, 3)
            cell_grad = flat[off:].view(T, 7)
    return vertices_grad, cell_grad


def vertex_backward(indices, vertices, cam, tiles_touched, grad_vs, grad_cc):
    lib = _lib.load()
    dev = vertices.device
    T, V = indices.shape[0], vertices.shape[0]
    with torch.cuda.device(dev):
        vertices_grad = torch.empty((V, 3), dtype=torch.float32, device=dev)
        _lib.check(lib.rm_vertex_backward(_ptr(indices), _ptr(vertices), T, V, cam.ref, _ptr(tiles_touched),
                                          _ptr(grad_vs), _ptr(grad_cc), _ptr(vertices_grad), _stream(dev)))
    return vertices_grad


def tet_err(sorted_idx, tile_ranges, records, cam, pixel_err, ssim_err, n_tets):
    """Densification statistics: (tet_err[T,16] f32, tet_count[T,2] i32)."""
    lib = _lib.load()
    dev = records.device
    with torch.cuda.device(dev):
        err = torch.empty((n_tets, 16), dtype=torch.float32, device=dev)
        cnt = torch.empty((n_tets, 2), dtype=torch.int32, device=dev)
        if _lib.bounds_checked():
            _lib.set_extents(list=sorted_idx.shape[0], tets=n_tets)
        _lib.check(lib.rm_tet_err(_ptr(sorted_idx), _ptr(tile_ranges), _ptr(records), cam.ref, _ptr(pixel_err),
                                  _ptr(ssim_err), n_tets, _ptr(err), _ptr(cnt), _stream(dev)))
    return err, cnt
