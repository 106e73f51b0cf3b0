"""The quick decision which texel-views a bake reads (csrc/projection.cuh: project_gate) against the projection's tests
in double precision, and the tiled order of the atlas (AtlasTiles) against the linear one.

Texels are placed at chosen distances from the facing limit and the clip volume's sides, some inside the margins where
the exact tests have to take over. The exact tests' own roundings (dot products of four fp32 terms: under 5 * 2^-24 of
the terms' magnitudes) leave texels within 2e-6 of a limit undecided; all others must agree."""
import ctypes as C

import numpy as np
import pytest
import torch

from photara_drender_gb300 import TextureBaker, _native
from photara_drender_gb300 import synthetic as S
from photara_drender_gb300.baking import ProjectionViewC
from photara_drender_gb300.rasterizer import _ptr

pytestmark = pytest.mark.gpu

VIEWPORTS = [(0, 0, 40, 30), (5.5, -3.25, 20, 11), (1e6, 0, 40, 30), (-700.0, 3.0, 50, 2.5)]


def decide(mat, cam, limit, p, n):
    """(inside, decided) in double precision."""
    M, p, n = mat.astype(np.float64), p.astype(np.float64), n.astype(np.float64)
    n = n / np.linalg.norm(n, axis=1, keepdims=True)
    c = p @ M[:, :3].T + M[:, 3]
    scale = np.abs(p) @ np.abs(M[:, :3]).max(0) + np.abs(M[:, 3]).max()
    v = cam.astype(np.float64) - p
    cosv = (n * v).sum(1) / np.linalg.norm(v, axis=1)
    gap = c[:, 3] - np.abs(c[:, :3]).max(1)
    return (gap > 0) & (cosv > limit), (np.abs(gap) > 2e-6 * scale) & (np.abs(cosv - limit) > 2e-6)


@pytest.mark.parametrize("shape,views", [((61, 37), 3), ((9, 16), 33), ((40, 15), 2), ((1, 130), 4), ((33, 1), 1)])
def test_gate_and_tiles(shape, views):
    baker = TextureBaker(0)
    dev = baker.context.device
    rng = np.random.default_rng(shape[0] * 64 + views)
    h, w = shape
    N = h * w
    mats, eyes = S.orbit_cameras(max(views, 2))
    mats, eyes = mats[:views], eyes[:views].astype(np.float32)
    limit = np.float32(0.25)
    # positions on clip-volume sides and normals at the facing limit of a random view, at distances 0 .. 1e-1
    k = rng.integers(0, views, N)
    inv = np.linalg.inv(mats.astype(np.float64))
    ndc = rng.uniform(-0.9, 0.9, (N, 3))
    step = rng.choice([1e-1, 1e-3, 1e-4, 3e-5, 1e-5, 4e-6, 0.0], (2, N)) * rng.choice([-1, 1], (2, N))
    side = rng.random(N) < 0.5
    axis = rng.integers(0, 2, N)
    ndc[side, axis[side]] = (rng.choice([-1.0, 1.0], N) * (1.0 + step[0]))[side]
    clip = np.concatenate([ndc, np.ones((N, 1))], 1)
    p = np.einsum("nij,nj->ni", inv[k], clip)
    p = (p[:, :3] / p[:, 3:]).astype(np.float32)
    v = eyes[k].astype(np.float64) - p
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    t = np.cross(v, rng.normal(size=(N, 3)))
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    c = np.clip(np.where(rng.random(N) < 0.5, limit + step[1], rng.uniform(-1, 1, N)), -1, 1)[:, None]
    nrm = ((c * v + np.sqrt(1 - c * c) * t) * rng.uniform(0.5, 2.0, (N, 1))).astype(np.float32)
    raster = np.zeros((h, w, 4), np.float32)
    raster.reshape(-1, 4)[:, 3] = rng.integers(0, 5, N) > 0
    d = {n: torch.tensor(x, device=dev) for n, x in dict(p=p, n=nrm, r=raster).items()}
    # a triangle far away: no ray meets it, so a bit is set exactly where the projection's tests pass
    tri = torch.tensor([[50.0, 50, 50], [51, 50, 50], [50, 51, 50]], device=dev)
    idx = torch.tensor([[0, 1, 2]], dtype=torch.int32, device=dev)
    image = torch.ones((30, 40, 3), device=dev)
    table = (ProjectionViewC * views)()
    for q in range(views):
        row = table[q]
        row.world_to_clip[:] = [float(x) for x in mats[q].reshape(16)]
        row.camera_position[:] = [float(x) for x in eyes[q]]
        row.weight, row.min_view_cosine = 1.0, float(limit)
        row.viewport[:] = VIEWPORTS[q % len(VIEWPORTS)]
        row.height, row.width, row.channel_count = 30, 40, 3
        row.image = image.data_ptr()
    tab = torch.frombuffer(bytearray(bytes(table)), dtype=torch.uint8).to(dev)
    s = baker.context.stream()
    nb, ns = C.c_size_t(), C.c_size_t()
    _native.call("pdr_bvh_sizes", 1, C.byref(nb), C.byref(ns))
    bvh = torch.empty(nb.value, dtype=torch.uint8, device=dev)
    scratch = torch.empty(ns.value, dtype=torch.uint8, device=dev)
    _native.call("pdr_bvh_build", _ptr(tri), 3, _ptr(idx), 1, _ptr(bvh), nb.value, _ptr(scratch), ns.value, s)
    results = []
    for width in (0, w):
        bits = torch.full((N, (views + 31) // 32), -1, dtype=torch.int32, device=dev)
        _native.call("pdr_ray_visibility_atlas", _ptr(bvh), 1, _ptr(d["p"]), _ptr(d["n"]), _ptr(d["r"]), N, width,
                     _ptr(tab), views, 1e-4, _ptr(bits), s)
        outs = [bits]
        for mode, vis in ((2, None), (2, _ptr(bits))):
            color = torch.full((N, 4), 7.0, device=dev)
            conf, valid, cov = (torch.full((N,), 7.0, device=dev) for _ in range(3))
            src, faces = (torch.full((N,), 7, dtype=torch.int32, device=dev) for _ in range(2))
            _native.call("pdr_project_views_atlas", _ptr(d["p"]), _ptr(d["n"]), _ptr(d["r"]), N, width, _ptr(tab), views,
                         1, 1, mode, vis, _ptr(color), _ptr(conf), _ptr(src), _ptr(valid), _ptr(cov), _ptr(faces), s)
            outs += [color, conf, src, valid, cov, faces]
        results.append([o.cpu().numpy() for o in outs])
    for a, b in zip(*results):
        assert np.array_equal(a, b)
    covered = raster.reshape(-1, 4)[:, 3] != 0
    bits, valid, seen = results[0][0].view(np.uint32), results[0][4], np.zeros(N, bool)
    all_decided = covered.copy()
    for q in range(views):
        inside, decided = decide(mats[q], eyes[q], float(limit), p, nrm)
        # a viewport far from the origin rounds pixel positions to its own step
        vp = np.array(VIEWPORTS[q % len(VIEWPORTS)], np.float64)
        c4 = p.astype(np.float64) @ mats[q][:, :3].T.astype(np.float64) + mats[q][:, 3]
        edge = np.abs(1 - np.abs(c4[:, :2] / c4[:, 3:])) * 0.5 * vp[2:]
        decided &= (edge > 2 * np.spacing((np.abs(vp[:2]) + vp[2:]).astype(np.float32))).all(1)
        got = (bits[:, q // 32] >> np.uint32(q % 32)) & 1
        ok = decided & covered
        assert np.array_equal(got[ok], inside[ok].astype(np.uint32)), q
        seen |= inside
        all_decided &= decided
    assert not bits[~covered].any()
    assert np.array_equal(valid[all_decided] != 0, seen[all_decided])


@pytest.mark.parametrize("channels,offset", [(3, 0), (4, 0), (4, 1)])
@pytest.mark.parametrize("pcf", [0, 1, 2, 4])
def test_inner_taps(channels, offset, pcf):
    """Shadow-map and photograph taps inside and across the borders of a view, at every radius, and of images whose
    rows are not 16-byte aligned, against the oracle's bake, bit for bit."""
    from oracle import api
    from tests.gpu_util import same_bits

    baker = TextureBaker(0)
    pos3, nrm, uv, idx, _, _ = S.displaced_sphere(2000, seed=pcf, amplitude=0.15, atlas_size=64)
    mats, eyes = S.orbit_cameras(3, fov_y_deg=30.0)  # the surface reaches past the views' borders
    rng = np.random.default_rng(9)
    images = [rng.uniform(size=(48, 40, channels)).astype(np.float32) for _ in range(3)]
    held = []
    for im in images:
        flat = torch.zeros(im.size + offset, device=baker.context.device)
        flat[offset:] = torch.tensor(im.reshape(-1), device=flat.device)
        held.append(flat[offset:].view(im.shape))
    out = baker.bake_output(pos3, nrm, uv, idx, held, mats, eyes, resolution=(64, 64), blend_mode="weighted_average",
                            visibility_mode="shadow_map", pcf_radius=pcf)
    color, conf, src, valid, _, _ = api.bake(pos3, nrm, uv, idx, images, mats, eyes, resolution=(64, 64),
                                             blend_mode="weighted_average", visibility_mode=0, pcf_radius=pcf)
    assert same_bits(np.asarray(out.color.cpu() if hasattr(out.color, "cpu") else out.color), color)
    assert same_bits(np.asarray(out.confidence.cpu() if hasattr(out.confidence, "cpu") else out.confidence), conf)
    assert valid.any()
