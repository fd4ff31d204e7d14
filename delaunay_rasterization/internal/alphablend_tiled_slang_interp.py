"""Stages 5-6 behind the reference's entry point
(delaunay_rasterization/internal/alphablend_tiled_slang_interp.py:10-112).

AlphaBlendTiledRender.apply(sorted_tetra_idx, tile_ranges, indices, vertices,
tet_density, render_grid, tcam, ray_jitter) -> (output_img[H,W,4],
distortion_img[H,W,5], tet_alive[T] bool); backward returns gradients for
`vertices` and `tet_density` only.  Any tile size is accepted (the reference
compiles 4x4 only).
"""
import torch

from delaunay_rasterization.internal.render_grid import RenderGrid  # noqa: F401  (re-exported by the reference)
from delaunay_rasterization.internal.tile_shader_slang import lookup_tiles_touched, vertex_and_tile_shader  # noqa: F401
from radiance_meshes_b200 import _lib, raster


def pack_ahead(bctx, indices, vertices, tet_density):
    """(camera, records) of a frame whose projection is enqueued, packed before its tile lists are built, for the last argument of
    AlphaBlendTiledRender.apply; None where the arguments are not such as that takes."""
    cam = bctx["cam"]
    packed = _lib.native().pack_ahead(indices, vertices, tet_density, cam.address, bctx["tiles_touched"])
    return None if packed is None else (cam, packed)


class AlphaBlendTiledRender(torch.autograd.Function):
    @staticmethod
    def forward(ctx, sorted_tetra_idx, tile_ranges, indices, vertices, tet_density, render_grid, tcam, ray_jitter, *extra):
        # extra: the reference's optional `device` argument, then what pack_ahead has returned for these arguments
        cam, packed = extra[1] if len(extra) > 1 and extra[1] is not None else (None, None)
        ctx.n_extra = len(extra)
        assert tet_density.shape[1] == 7, "cell values are (density, r, g, b, gx, gy, gz) per tet"
        if ray_jitter is not None:  # None: the pixel centres
            assert ray_jitter.shape == (render_grid.image_height, render_grid.image_width, 2)
            if ray_jitter.dtype != torch.float32 or not ray_jitter.is_contiguous():
                # once for both directions: the caller may refill a jitter that was copied as soon as this returns
                ray_jitter = ray_jitter.detach().float().contiguous()
        raster._require_cuda(vertices, "vertices")
        if cam is None:
            cam = raster.CameraArgs(tcam, vertices.device)
        assert cam.native.grid == (render_grid.grid_height, render_grid.grid_width)
        need_grad = vertices.requires_grad or tet_density.requires_grad
        out = _lib.native().blend_forward(sorted_tetra_idx, tile_ranges, indices, vertices, tet_density, cam.address,
                                          cam.native.zero_fill, ray_jitter, lookup_tiles_touched(sorted_tetra_idx),
                                          need_grad, packed)
        output_img, distortion_img, tet_alive, indices, verts, cell, records, n_contributors = out[:8]
        if need_grad:
            ctx.save_for_backward(sorted_tetra_idx, tile_ranges, indices, verts, cell, output_img, distortion_img,
                                  ray_jitter, n_contributors, records, *out[8:])
            ctx.cam = cam
        ctx.mark_non_differentiable(tet_alive)
        ctx.set_materialize_grads(False)  # a gradient that was not asked for is not filled with zeros
        return output_img, distortion_img, tet_alive

    @staticmethod
    def backward(ctx, grad_output_img, grad_distortion_img, grad_vert_alive):
        (sorted_tetra_idx, tile_ranges, indices, verts, cell, output_img, distortion_img, jitter, n_contributors,
         records, tet_flags, hit_counts, hit_ids, hit_masks) = ctx.saved_tensors
        if grad_output_img is None:
            grad_output_img = torch.zeros_like(output_img)
        if grad_distortion_img is None:
            grad_distortion_img = torch.zeros_like(distortion_img)
        vertices_grad, cell_grad = raster.backward(
            sorted_tetra_idx, tile_ranges, records, ctx.cam, jitter, output_img, distortion_img, n_contributors,
            (hit_counts, hit_ids, hit_masks, tet_flags), grad_output_img.float(), grad_distortion_img.float(), indices,
            verts, cell)
        return (None, None, None, vertices_grad, cell_grad, None, None, None) + (None,) * ctx.n_extra
