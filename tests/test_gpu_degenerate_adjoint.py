"""Attribute gradients of triangles with repeated vertices under non-finite upstream gradients: each distinct vertex
receives its accumulated weight times the gradient once, a repeated corner nothing, as in the oracle, bit for bit (one
pixel per triangle and triangles without common vertices, so that nothing is summed). A NaN's sign and payload are free."""
import numpy as np
import pytest

import photara_drender_gb300 as pdr
from oracle import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("attributes", [1, 3, 8, 9, 17])
def test_repeated_vertices_and_non_finite_gradients(attributes):
    rng = np.random.default_rng(attributes)
    corners = np.array([[0, 1, 2], [0, 0, 1], [0, 1, 0], [0, 1, 1], [0, 0, 0]])
    T = 60
    idx = (corners[np.arange(T) % 5] + 3 * np.arange(T)[:, None]).astype(np.uint32)
    raster = rng.uniform(0, 0.5, (4, 15, 4)).astype(np.float32)
    raster[..., 3] = rng.permutation(T).reshape(4, 15) + 1
    attrs = rng.uniform(size=(3 * T, attributes)).astype(np.float32)
    g = rng.normal(size=(4, 15, attributes)).astype(np.float32)
    g[rng.uniform(size=g.shape) < 0.3] = np.inf
    g[rng.uniform(size=g.shape) < 0.2] = -np.inf
    g[rng.uniform(size=g.shape) < 0.1] = np.nan
    got, got_r = pdr.Rasterizer().interpolate_backward(attrs, idx, raster, g)
    with np.errstate(all="ignore"):
        want, want_r = api.interpolate_backward(attrs, idx, raster, g)
    assert np.isinf(want).any()
    np.testing.assert_array_equal(got, want)  # equal values, NaN where NaN
    np.testing.assert_array_equal(got_r, want_r)
