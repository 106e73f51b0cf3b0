"""The visibility-buffer forward (pdr_render_direct) against the oracle and against the tile path
(pdr_bin_tiles + pdr_rasterize_forward), bit for bit: triangles of every scale, images smaller than a tile and
ragged ones, warps with one to 32 triangles, the queue of large triangles, several groups of views."""
import numpy as np
import pytest
import torch

import photara_drender_gb300 as pdr
from oracle import api
from photara_drender_gb300 import synthetic as S
from tests.gpu_util import same_bits

pytestmark = pytest.mark.gpu


def soup(rng, n):
    """Clip positions of n separate triangles from microscopic to larger than the image, with slivers, shared
    depths, vertices behind the eye and a few non-finite ones."""
    xy = rng.uniform(-1.5, 1.5, (n, 1, 2)) + rng.normal(size=(n, 3, 2)) * 10 ** rng.uniform(-5.5, 0.5, (n, 1, 1))
    sliver = rng.uniform(size=n) < 0.2
    xy[sliver, 2] = xy[sliver, :2].mean(1) + 1e-6 * rng.normal(size=(sliver.sum(), 2))
    w = rng.uniform(0.2, 2.2, (n, 3, 1))
    w[rng.uniform(size=w.shape) < 0.02] *= -1
    z = rng.choice([-0.5, 0.0, 0.25], size=(n, 1, 1))
    z = z + np.where(rng.uniform(size=(n, 1, 1)) < 0.5, 0, rng.normal(size=(n, 3, 1)))
    clip = np.concatenate([xy * w, z * w, w], -1).reshape(3 * n, 4).astype(np.float32)
    if n > 20:
        clip[5, 0], clip[22, 1], clip[40, 3] = np.nan, np.inf, np.inf
    return clip, np.arange(3 * n, dtype=np.uint32).reshape(n, 3)


@pytest.mark.parametrize("triangles,res,viewport,cull", [
    (1, (1, 1), None, "none"), (3, (7, 5), None, "none"), (40, (17, 33), None, "back"),
    (700, (96, 257), None, "front"), (700, (130, 70), (3.0, -2.0, 60.5, 131.25), "none"),
    (3000, (64, 1100), (-100.0, 10.0, 1300.0, 40.0), "none"), (150, (600, 500), None, "none")])
def test_direct_forward_matches_oracle(triangles, res, viewport, cull):
    rng = np.random.default_rng(triangles + res[0])
    clip, idx = soup(rng, triangles)
    want, want_d = api.rasterize_forward(clip, idx, res, ["none", "back", "front"].index(cull), viewport=viewport)
    got, got_d = pdr.Rasterizer().forward(clip, idx, res, cull, True, viewport)
    assert same_bits(got, want) and same_bits(got_d, want_d)


def test_direct_forward_in_groups_of_views():
    """70 views at 1024 x 1024 exceed one group's keys: views of the first and of the second group equal the
    same views rendered alone."""
    pos3, idx = S.icosphere(3)
    mats, _ = S.orbit_cameras(70)
    dev = torch.device("cuda", 0)
    clip = torch.tensor(S.clip_positions(pos3, mats), device=dev)
    tidx = torch.tensor(idx.astype(np.int32), device=dev)
    r = pdr.Rasterizer()
    raster, _ = r.forward(clip, tidx, (1024, 1024), output_barycentric_derivatives=False)
    for k in (0, 63, 64, 69):
        one, _ = r.forward(clip[k], tidx, (1024, 1024), output_barycentric_derivatives=False)
        assert torch.equal(raster[k].view(torch.int32), one.view(torch.int32)), k


@pytest.mark.parametrize("attributes", [0, 1, 2, 4, 5, 8])
def test_direct_shading_matches_separate_kernels(attributes):
    rng = np.random.default_rng(attributes)
    pos3, idx = S.icosphere(4)
    mats, _ = S.orbit_cameras(2)
    dev = torch.device("cuda", 0)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=dev)  # noqa: E731
    clip, uv = t(S.clip_positions(pos3, mats)), t(S.spherical_uv(pos3) * 1.3 - 0.2)
    tex, tidx = t(rng.uniform(size=(37, 50, 4))), torch.tensor(idx.astype(np.int32), device=dev)
    attrs = t(rng.uniform(size=(pos3.shape[0], attributes))) if attributes else None
    r = pdr.Rasterizer()
    o = pdr.render(clip, tidx, (75, 101), rasterizer=r, vertex_attributes=attrs, vertex_uv=uv, texture=tex,
                   address_mode="mirror")
    raster, deriv = r.forward(clip, tidx, (75, 101))
    u = r.interpolate_forward(uv, tidx, raster)
    pairs = [(o.raster, raster), (o.derivatives, deriv), (o.uv, u),
             (o.sampled, r.texture_forward(tex, u, raster, "mirror"))]
    if attributes:
        pairs.append((o.interpolated, r.interpolate_forward(attrs, tidx, raster)))
    for a, b in pairs:
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
