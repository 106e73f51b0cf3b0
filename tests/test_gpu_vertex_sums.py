"""Vertex gradients summed per warp and triangle (csrc/vertex_sums.cuh) in the separate adjoints: attribute counts on
both sides of the compiled ones, images whose last warp is partial, degenerate triangles with repeated vertices, and
meshes from one triangle per pixel to one for all, against the oracle's FP64 sums."""
import numpy as np
import pytest

import photara_drender_gb300 as pdr
from oracle import api
from photara_drender_gb300 import synthetic as S
from tests.gpu_util import grad_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("attributes", [1, 2, 5, 8, 9, 17])
@pytest.mark.parametrize("subdivisions,res", [(0, (33, 31)), (4, (40, 57))])
def test_separate_adjoints_match_oracle(attributes, subdivisions, res):
    rng = np.random.default_rng(attributes)
    pos3, idx = S.icosphere(subdivisions)
    idx[::7, 2] = idx[::7, 0]  # repeated vertices: never covered, but a raster may name them
    mats, _ = S.orbit_cameras(1)
    clip = S.clip_positions(pos3, mats)[0]
    raster, _ = api.rasterize_forward(clip, idx, res)
    named = rng.uniform(size=res) < 0.1
    raster[..., 3] = np.where(named & (raster[..., 3] > 0), 1 + 7 * rng.integers(0, len(idx) // 7, res), raster[..., 3])
    attrs = rng.uniform(size=(len(pos3), attributes)).astype(np.float32)
    g = rng.normal(size=res + (attributes,)).astype(np.float32)
    r = pdr.Rasterizer()
    ga, gr = r.interpolate_backward(attrs, idx, raster, g)
    want, want_r = api.interpolate_backward(attrs, idx, raster, g)
    exact = api.interpolate_backward(attrs, idx, raster, g, f64=True)[0]
    terms = api.interpolate_backward(attrs, idx, raster, g, f64=True, abs_terms=True)[0]
    grad_check(ga, want, exact, terms, name="attributes")
    assert np.array_equal(gr.view(np.uint32), want_r.view(np.uint32))
    grad_check(r.backward(clip, idx, raster, want_r), api.rasterize_backward(clip, idx, raster, want_r),
               api.rasterize_backward(clip, idx, raster, want_r, f64=True),
               api.rasterize_backward(clip, idx, raster, want_r, f64=True, abs_terms=True), name="clip")
