"""The adjoint's pixel bounds (render_bwd_tile.cuh: visited) for clip positions of every magnitude: pixels of a raster
that names a triangle outside its bounds pass no gradient, as in the oracle, also where the quotients' fast form is not
defined (w from 2^126 on)."""
import numpy as np
import pytest

import photara_drender_gb300 as pdr
from oracle import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1e-6, 1.0, 1e20, 8.4e37, 8.6e37, 1e38, 1.6e38])
@pytest.mark.parametrize("place", [(1.3, 0.0), (-1.6, 0.1), (0.0, 1.4), (0.0, -1.5)])
def test_pixels_outside_a_triangles_bounds(w, place):
    corners = np.array([[-0.1, -0.1], [0.1, -0.1], [0.0, 0.1]]) + place  # NDC: past one side of the image
    clip = np.concatenate([corners * w, np.zeros((3, 1)), np.full((3, 1), w)], 1).astype(np.float32)
    idx = np.array([[0, 1, 2]], np.uint32)
    raster = np.zeros((5, 5, 4), np.float32)
    raster[..., :2], raster[..., 3] = 0.25, 1.0
    g = np.random.default_rng(0).normal(size=(5, 5, 4)).astype(np.float32)
    want = api.rasterize_backward(clip, idx, raster, g)
    assert not want.any()
    assert not np.asarray(pdr.Rasterizer().backward(clip, idx, raster, g)).any()
