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


@pytest.mark.parametrize("address", ["clamp", "wrap"])
def test_sorted_tiles_match_separate_kernels(address):
    """Views of a texture above L2's size, sampled densely enough that the shading and the adjoint take their tiles
    by what they sample: images bit for bit, gradients up to the summation order of the atomics."""
    rng = np.random.default_rng(3)
    pos3, idx = S.icosphere(5)
    mats, _ = S.orbit_cameras(6)
    dev = torch.device("cuda", 0)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=dev, requires_grad=True)  # noqa: E731
    inputs = [S.clip_positions(pos3, mats), rng.uniform(size=(len(pos3), 3)), S.spherical_uv(pos3) * 1.4 - 0.2]
    tidx = torch.tensor(idx.astype(np.int32), device=dev)
    texture = torch.rand((2900, 2900, 4), device=dev, generator=torch.Generator(dev).manual_seed(1))
    res = (870, 1013)  # ragged in both directions
    g_attr, g_tex = torch.randn((6,) + res + (3,), device=dev), torch.randn((6,) + res + (4,), device=dev)
    r = pdr.Rasterizer()
    results = []
    for fused in (True, False):
        clip, attrs, uv = (t(a) for a in inputs)
        tex = texture.clone().requires_grad_(True)
        if fused:
            raster, _, a, u, s = pdr.render(clip, tidx, res, rasterizer=r, vertex_attributes=attrs, vertex_uv=uv,
                                            texture=tex, address_mode=address)
        else:
            raster, _ = pdr.rasterize(clip, tidx, res, rasterizer=r)
            a, u = (pdr.interpolate(x, raster, tidx, rasterizer=r) for x in (attrs, uv))
            s = pdr.texture(tex, u, raster, rasterizer=r, address_mode=address)
        torch.autograd.backward([a, s], [g_attr, g_tex])
        results.append(([raster, a, u, s], [clip.grad, attrs.grad, uv.grad, tex.grad]))
    for x, y in zip(results[0][0], results[1][0]):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))
    for x, y in zip(results[0][1], results[1][1]):
        assert float((x - y).abs().max()) <= 1e-4 * float(y.abs().max()) + 1e-7


def test_batch_in_groups_of_jobs():
    """A batch whose keys exceed one group: views on both sides of the border equal single renders."""
    from photara_drender_gb300.batch import BatchMesh, MeshBatch

    dev = torch.device("cuda", 0)
    r = pdr.Rasterizer()
    meshes = []
    for sub, views, side in ((2, 3, 70), (3, 66, 1024)):
        pos3, idx = S.icosphere(sub)
        mats, _ = S.orbit_cameras(views)
        meshes.append(BatchMesh(torch.tensor(S.clip_positions(pos3, mats), device=dev),
                                torch.tensor(idx.astype(np.int32), device=dev), side, side))
    MeshBatch(r, meshes).forward()
    for m, views in zip(meshes, ((0, 2), (0, 62, 63, 64, 65))):
        for k in views:
            one, d = r.forward(m.clip[k], m.indices, (m.height, m.width))
            assert torch.equal(m.outputs["raster"][k].view(torch.int32), one.view(torch.int32)), k
            assert torch.equal(m.outputs["deriv"][k].view(torch.int32), d.view(torch.int32)), k


@pytest.mark.parametrize("capture", [False, True])
def test_pipeline_through_the_visibility_buffer(capture):
    """RenderFwdBwd(direct=True) gives the images of the tile lists bit for bit and the same gradients up to the order
    of their sums, as launches and as a replayed graph."""
    from photara_drender_gb300.pipeline import RenderFwdBwd

    rng = np.random.default_rng(3)
    pos3, idx = S.icosphere(4)
    mats, _ = S.orbit_cameras(3)
    dev = torch.device("cuda", 0)
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device=dev)  # noqa: E731
    V, H, W = pos3.shape[0], 75, 101
    args = [t(S.clip_positions(pos3, mats)), t(rng.uniform(size=(V, 3))), t(S.spherical_uv(pos3)),
            t(rng.uniform(size=(64, 48, 4))), t(rng.normal(size=(3, H, W, 3))), t(rng.normal(size=(3, H, W, 4)))]
    tidx = torch.tensor(idx.astype(np.int32), device=dev)
    pipes = [RenderFwdBwd(pdr.Rasterizer(), tidx, V, 3, H, W, 3, (64, 48, 4), direct=d,
                          viewports=[None, (5.0, -3.0, 90.0, 70.0), None]) for d in (False, True)]
    pipes[0].step(*args)
    if capture:
        graph = pipes[1].capture(*args)
        for k in ("raster", "sampled", "grad_clip", "grad_tex"):
            getattr(pipes[1], k).fill_(9.0)
        graph.replay()
    else:
        pipes[1].step(*args)
    torch.cuda.synchronize()
    for k in ("raster", "deriv", "attr_out", "uv", "sampled"):
        assert torch.equal(*(getattr(p, k).view(torch.int32) for p in pipes)), k
    for k in ("grad_clip", "grad_attr", "grad_uv_attr", "grad_tex"):
        a, b = (getattr(p, k) for p in pipes)
        assert float((a - b).abs().max()) <= 1e-5 * float(a.abs().max()), k
    assert pipes[1].check_capacity() == 0 and pipes[1].autotune(*args[:4]) == {} and pipes[1].kernels_per_step() == 5
