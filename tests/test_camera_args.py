"""Cameras as the host path takes them (no GPU: the camera's arrays may be in host memory as long as nothing is launched)."""
import collections
import types

import numpy as np
import pytest
import torch

from radiance_meshes_b200 import raster, scenes


def tcam(**kw):
    return dict(scenes.make_tcam(scenes.look_at((0.3, 0.2, 2.5)), 40, 52, 60.0, tile=4, min_t=0.1), **kw)


class Subscripts:
    """Neither a dict nor a Mapping: what a camera is asked for, and no more."""

    def __init__(self, values):
        self.values = values

    def __getitem__(self, key):
        return self.values[key]

    def get(self, key, default=None):
        return self.values.get(key, default)


@pytest.mark.parametrize("kind", [dict, collections.OrderedDict, collections.UserDict, types.MappingProxyType,
                                  lambda d: collections.ChainMap({}, d), Subscripts])
@pytest.mark.parametrize("extra,rows,only", [({}, (0, 10), False), (dict(tile_rows=(2, 7)), (2, 7), False),
                                             (dict(tile_rows=[1, 3], band_rows_only=True), (1, 3), True),
                                             (dict(band_rows_only=np.bool_(False)), (0, 10), False)])
def test_any_kind_of_dictionary(cuda_lib, kind, extra, rows, only):
    cam = raster.CameraArgs(kind(tcam(**extra)), torch.device("cpu"))
    c = cam.c
    assert (c.tile_row_begin, c.tile_row_end, cam.band_rows_only) == (*rows, only)
    assert (c.image_height, c.image_width, c.grid_height, c.grid_width, c.tile_width) == (40, 52, 10, 13, 4)
    assert cam.native.grid == (10, 13) and cam.native.zero_fill == (rows != (0, 10) and not only)
    assert abs(c.min_t - 0.1) < 1e-7


def test_a_missing_field_is_named(cuda_lib):
    d = tcam()
    del d["tile_width"]
    with pytest.raises(KeyError, match="tile_width"):
        raster.CameraArgs(d, torch.device("cpu"))


def test_rows_given_with_the_call_come_first(cuda_lib):
    cam = raster.CameraArgs(tcam(tile_rows=(2, 7)), torch.device("cpu"), tile_rows=(3, 4))
    assert (cam.c.tile_row_begin, cam.c.tile_row_end) == (3, 4)
