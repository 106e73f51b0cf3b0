"""Performance cases of the framework's public calls, with what a pass of each cannot do without.

The workloads are those of the benchmark table and of the tests: fused and separate differentiable
rendering, texture baking in both visibility modes, atlas refinement, uneven mesh batches and atlas
padding. Meshes are displaced cube spheres with six charts packed 3 x 2 (the benchmark's sphere, made on
the GPU), cameras look at the origin from Fibonacci directions. `exact` restates each path in float64
torch operations.
"""
import math

import numpy as np
import torch

DEV = "cuda"
F64 = torch.float64
ADDRESS = {"clamp": 0, "wrap": 1, "mirror": 2}


def listed():
    return [
        # one small training step on a preview image: latency and launches are the cost
        dict(name="render_1x256", kind="render", n=10, views=1, h=256, w=256, attrs=3, tex_h=256, tex_w=256,
             address="clamp", cull="none", deferred=False),
        # the benchmark's small configuration: about 5k triangles, 8 views at 512 x 512, 1024 x 1024 texture
        dict(name="render_8x512", kind="render", n=21, views=8, h=512, w=512, attrs=3, tex_h=1024, tex_w=1024,
             address="clamp", cull="none", deferred=False),
        # the benchmark's headline: 200k triangles, 64 views at 1024 x 1024, 4096 x 4096 atlas, no host waits
        dict(name="render_64x1024", kind="render", n=129, views=64, h=1024, w=1024, attrs=3, tex_h=4096, tex_w=4096,
             address="clamp", cull="none", deferred=True),
        # rasterize -> interpolate -> texture as separate calls (the reference's own interface), one photograph
        # of an odd size, an RGB texture that tiles
        dict(name="chain_1x637x479", kind="chain", n=41, views=1, h=479, w=637, attrs=3, tex_h=700, tex_w=1000,
             channels=3, address="wrap", cull="none"),
        # the separate calls over several views of a dense mesh with back faces culled
        dict(name="chain_8x1024", kind="chain", n=129, views=8, h=1024, w=1024, attrs=5, tex_h=2048, tex_w=2048,
             channels=4, address="clamp", cull="back"),
        # texture bake with shadow maps from 24 photographs
        dict(name="bake_shadow_2048", kind="bake", n=129, views=24, h=1024, w=1024, channels=3, atlas_h=2048,
             atlas_w=2048, visibility="shadow_map", blend="weighted_average", pcf=1, masks=False),
        # texture bake with the default ray-query visibility, RGBA photographs with masks, a ragged atlas
        dict(name="bake_ray_2000x1500", kind="bake", n=129, views=16, h=768, w=1024, channels=4, atlas_h=1500,
             atlas_w=2000, visibility="ray_query", blend="weighted_average", pcf=1, masks=True),
        # a short refinement of a small atlas with the default options and the seam polish
        dict(name="refine_512", kind="refine", n=21, views=6, h=240, w=320, atlas_h=512, atlas_w=512, steps=60, batch=4,
             tv=0.0, pairs=1200, polish=10),
        # the benchmark's refinement size: 500k triangles, 2048 x 1536 views, 4096 x 4096 atlas, total variation
        dict(name="refine_4096_tv", kind="refine", n=204, views=8, h=1536, w=2048, atlas_h=4096, atlas_w=4096,
             steps=100, batch=4, tv=1e-2, pairs=20000, polish=5),
        # six meshes of uneven size in one batch, 8 attributes
        dict(name="batch_6", kind="batch", meshes=6, n_min=29, n_max=204, views_max=12, side_max=1024, attrs=8,
             tex=2048),
        # padding of a baked atlas: 4-texel gutters and every unobserved covered texel
        dict(name="pad_4096_fill", kind="pad", atlas_h=4096, atlas_w=4096, channels=4, margin=4, fill=True, distance=0),
        # gutters alone on a ragged RGB atlas
        dict(name="pad_1400x1000", kind="pad", atlas_h=1000, atlas_w=1400, channels=3, margin=8, fill=False,
             distance=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "chain", "chain", "bake", "refine", "batch", "pad"])
    if kind in ("render", "chain"):
        views = _log(rng, 1, 16)
        side = _log(rng, 160, 1280)
        c = dict(kind=kind, n=_log(rng, 8, 180), views=views, h=side, w=max(64, int(side * rng.uniform(0.6, 1.6))),
                 attrs=rng.randint(1, 8), tex_h=_log(rng, 200, 3000), tex_w=_log(rng, 200, 3000),
                 address=rng.choice(["clamp", "wrap", "mirror"]), cull=rng.choice(["none", "none", "back"]))
        if kind == "render":
            c["deferred"] = rng.random() < 0.5
        else:
            c["channels"] = rng.choice([1, 3, 4])
        return c
    if kind == "bake":
        return dict(kind=kind, n=_log(rng, 20, 150), views=_log(rng, 3, 24), h=_log(rng, 300, 1024),
                    w=_log(rng, 300, 1024), channels=rng.choice([3, 4]), atlas_h=_log(rng, 400, 2048),
                    atlas_w=_log(rng, 400, 2048), visibility=rng.choice(["shadow_map", "ray_query"]),
                    blend=rng.choice(["weighted_average", "best_view", "softmax"]), pcf=rng.randint(0, 2),
                    masks=rng.random() < 0.5)
    if kind == "refine":
        tv = rng.random() < 0.5
        return dict(kind=kind, n=_log(rng, 15, 150), views=rng.randint(2, 8), h=_log(rng, 200, 1200),
                    w=_log(rng, 200, 1600), atlas_h=_log(rng, 300, 3000), atlas_w=_log(rng, 300, 3000),
                    steps=_log(rng, 10, 80), batch=rng.randint(1, 4), tv=1e-2 if tv else 0.0,
                    pairs=rng.choice([0, 900, 7000]), polish=rng.randint(2, 10))
    if kind == "batch":
        return dict(kind=kind, meshes=rng.randint(2, 6), n_min=_log(rng, 10, 40), n_max=_log(rng, 60, 180),
                    views_max=rng.randint(3, 10), side_max=_log(rng, 300, 1024), attrs=rng.choice([1, 3, 8]),
                    tex=_log(rng, 300, 2048))
    return dict(kind="pad", atlas_h=_log(rng, 200, 4096), atlas_w=_log(rng, 200, 4096), channels=rng.choice([3, 4]),
                margin=rng.randint(1, 16), fill=rng.random() < 0.5, distance=rng.choice([0, 0, 24]))


# ---- scenes -------------------------------------------------------------------------------------------

def _rng(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + salt)
    return g


def _mesh(n, seed):
    """Cube sphere of 12 n^2 triangles with a radial displacement r = 1 + 0.05 sum_8 sin(k.d + phi) / 8, one
    chart per cube face: positions, normals, uv (float32) and indices (int32)."""
    t = torch.linspace(-1, 1, n + 1, device=DEV, dtype=F64)
    b, a = torch.meshgrid(t, t, indexing="ij")
    one = torch.ones_like(a)
    faces = [(one, b, -a), (-one, b, a), (a, one, -b), (a, -one, b), (a, b, one), (-a, b, -one)]
    d = torch.stack([torch.stack(f, -1).reshape(-1, 3) for f in faces])
    d = d / d.norm(dim=-1, keepdim=True)
    g = _rng(seed, 1)
    k = torch.randn((8, 3), generator=g, device=DEV, dtype=F64) * 3.0
    phase = torch.rand(8, generator=g, device=DEV, dtype=F64) * (2 * math.pi)
    arg = d @ k.T + phase
    pos = d * (1.0 + 0.05 * torch.sin(arg).sum(-1, keepdim=True) / 8.0)
    # gradient of the radius gives the normal: n ~ r d - grad_tangent(r)
    grad = 0.05 / 8.0 * torch.cos(arg) @ k
    tangent = grad - (grad * d).sum(-1, keepdim=True) * d
    nrm = d * (1.0 + 0.05 * torch.sin(arg).sum(-1, keepdim=True) / 8.0) - tangent
    nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    f = torch.arange(6, device=DEV)
    cell = torch.stack([f % 3, f // 3], -1).to(F64)[:, None]
    local = torch.stack([a.reshape(-1), b.reshape(-1)], -1)[None] * 0.5 + 0.5
    size = torch.tensor([1 / 3, 1 / 2], device=DEV, dtype=F64)
    uv = (cell + 0.02 + local * 0.96) * size
    q = torch.arange(n, device=DEV)
    v0 = (q[:, None] * (n + 1) + q[None]).reshape(-1)
    quad = torch.stack([v0, v0 + 1, v0 + n + 2, v0, v0 + n + 2, v0 + n + 1], -1).reshape(-1, 3)
    idx = (quad[None] + (f * (n + 1) ** 2)[:, None, None]).reshape(-1, 3)
    return (pos.reshape(-1, 3).float(), nrm.reshape(-1, 3).float(), uv.reshape(-1, 2).float().contiguous(),
            idx.to(torch.int32).contiguous())


def _cameras(count, aspect, radius=3.0, fov=45.0, near=0.1, far=10.0):
    """world_to_clip [count, 4, 4] and eyes [count, 3] (float32 NumPy), looking at the origin."""
    i = np.arange(count) + 0.5
    phi, theta = np.arccos(1 - 2 * i / count), math.pi * (1 + 5 ** 0.5) * i
    eyes = radius * np.stack([np.cos(theta) * np.sin(phi), np.cos(phi), np.sin(theta) * np.sin(phi)], 1)
    mats = []
    f = 1.0 / math.tan(math.radians(fov) / 2)
    for e in eyes:
        z = -e / np.linalg.norm(e)
        x = np.cross([0.0, 1.0, 0.0] if abs(z[1]) < 0.99 else [1.0, 0.0, 0.0], z)
        x /= np.linalg.norm(x)
        R = np.stack([x, np.cross(z, x), z])
        t = -R @ e
        M = np.zeros((4, 4))
        M[0, :3], M[0, 3] = f / aspect * R[0], f / aspect * t[0]
        M[1, :3], M[1, 3] = f * R[1], f * t[1]
        s = (far + near) / (far - near)
        M[2, :3], M[2, 3] = s * R[2], s * t[2] - 2 * far * near / (far - near)
        M[3, :3], M[3, 3] = R[2], t[2]
        mats.append(M)
    return np.stack(mats).astype(np.float32), eyes.astype(np.float32)


def _clip(pos, mats):
    p = torch.cat([pos.to(F64), torch.ones_like(pos[:, :1], dtype=F64)], 1)
    return (p @ torch.from_numpy(mats).to(DEV, F64).transpose(1, 2)).float().contiguous()


def _image(g, h, w, c, cells=24, noise=0.01):
    """Smooth noise in [0, 1] with a little pixel noise: a photograph or an atlas."""
    low = torch.rand((1, c, cells, cells), generator=g, device=DEV)
    img = torch.nn.functional.interpolate(low, size=(h, w), mode="bicubic", align_corners=True)[0].permute(1, 2, 0)
    img = img + noise * torch.randn((h, w, c), generator=g, device=DEV)
    return img.clamp(0, 1).contiguous()


def _render_scene(c, seed):
    pos, _, uv, idx = _mesh(c["n"], seed)
    mats, _ = _cameras(c["views"], c["w"] / c["h"])
    g = _rng(seed, 2)
    ch = c.get("channels", 4)
    shape = (c["views"], c["h"], c["w"])
    s = dict(case=c, idx=idx, clip=_clip(pos, mats), uv=uv,
             attrs=torch.rand((pos.shape[0], c["attrs"]), generator=g, device=DEV),
             tex=torch.rand((c["tex_h"], c["tex_w"], ch), generator=g, device=DEV),
             g_attr=torch.randn(shape + (c["attrs"],), generator=g, device=DEV),
             g_tex=torch.randn(shape + (ch,), generator=g, device=DEV))
    if c["views"] == 1:  # the unbatched forms
        for k in ("clip", "g_attr", "g_tex"):
            s[k] = s[k][0]
    return s


def _photo_scene(c, seed):
    pos, nrm, uv, idx = _mesh(c["n"], seed)
    mats, eyes = _cameras(c["views"], c["w"] / c["h"])
    g = _rng(seed, 3)
    images = [_image(g, c["h"], c["w"], c.get("channels", 3)) for _ in range(c["views"])]
    for im in images:
        if im.shape[2] == 4:
            im[..., 3] = 1.0
    masks = None
    if c.get("masks", True):
        masks = [(_image(g, c["h"], c["w"], 1, noise=0.0)[..., 0] > 0.25).float() for _ in range(c["views"])]
    return dict(case=c, pos=pos, nrm=nrm, uv=uv, idx=idx, mats=mats, eyes=eyes, images=images, masks=masks)


def _batch_sizes(c):
    """(n, views, h, w, texture side) of each mesh: triangle counts spread over the logarithm of the range."""
    out = []
    for k in range(c["meshes"]):
        t = k / max(c["meshes"] - 1, 1)
        n = int(round(c["n_min"] * (c["n_max"] / c["n_min"]) ** t))
        side = max(64, c["side_max"] >> (k % 2))
        out.append((n, 2 + (k * 5) % c["views_max"], side, side if k % 3 else side * 4 // 3,
                    max(64, c["tex"] >> (k % 3))))
    return out


def _batch_scenes(c, seed):
    return [_render_scene(dict(n=n, views=v, h=h, w=w, attrs=c["attrs"], tex_h=t, tex_w=t), seed + 1000 * k)
            for k, (n, v, h, w, t) in enumerate(_batch_sizes(c))]


def _pad_scene(c, seed):
    """A 3 x 2 chart atlas with gutters, part of the covered texels unobserved (one contiguous region per
    smooth blob), as a bake leaves it."""
    h, w = c["atlas_h"], c["atlas_w"]
    g = _rng(seed, 4)
    y = torch.arange(h, device=DEV, dtype=F64)[:, None] / h * 2 % 1
    x = torch.arange(w, device=DEV, dtype=F64)[None] / w * 3 % 1
    covered = (y > 0.02) & (y < 0.98) & (x > 0.02) & (x < 0.98)
    low = torch.rand((1, 1, 40, 40), generator=g, device=DEV)
    blobs = torch.nn.functional.interpolate(low, size=(h, w), mode="bicubic", align_corners=True)[0, 0]
    valid = covered & (blobs > 0.12)
    color = _image(g, h, w, c["channels"]) * valid[..., None]
    return dict(case=c, color=color.contiguous(), valid=valid.float(), covered=covered.float())


def _refine_extra(c, seed):
    g = _rng(seed, 5)
    init = _image(g, c["atlas_h"], c["atlas_w"], 3, noise=0.05)
    h, w = c["atlas_h"], c["atlas_w"]
    chart = torch.arange(h, device=DEV)[:, None] * 2 // h * 3 + torch.arange(w, device=DEV)[None] * 3 // w
    y = torch.arange(h, device=DEV, dtype=F64)[:, None] / h * 2 % 1
    x = torch.arange(w, device=DEV, dtype=F64)[None] / w * 3 % 1
    valid = (y > 0.02) & (y < 0.98) & (x > 0.02) & (x < 0.98)
    pairs = None
    if c["pairs"]:  # points along the charts' borders against points along the next chart's
        t = torch.rand(c["pairs"], generator=g, device=DEV)
        f = torch.randint(0, 5, (c["pairs"],), generator=g, device=DEV)
        a = torch.stack([(f % 3 + 0.02) / 3, (f // 3 + 0.02 + 0.96 * t) / 2], -1)
        b = torch.stack([((f + 1) % 3 + 0.02 + 0.96 * t) / 3, ((f + 1) // 3 + 0.98) / 2], -1)
        pairs = torch.stack([a, b], 1).float().contiguous()
    return init, chart.to(torch.int32).contiguous(), valid.float().contiguous(), pairs


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("render", "chain"):
        from photara_drender_gb300 import Rasterizer

        s = _render_scene(case, seed)
        s["rasterizer"] = Rasterizer()
        for k in ("clip", "attrs", "uv", "tex"):
            s[k].requires_grad_(True)
        return s
    if kind in ("bake", "refine"):
        from photara_drender_gb300 import TextureBaker

        s = _photo_scene(case, seed)
        s["baker"] = TextureBaker()
        if kind == "refine":
            s["init"], s["chart"], s["valid"], s["pairs"] = _refine_extra(case, seed)
        return s
    if kind == "batch":
        from photara_drender_gb300 import Rasterizer
        from photara_drender_gb300.batch import BatchMesh, MeshBatch

        meshes = []
        for s in _batch_scenes(case, seed):
            m = BatchMesh(s["clip"], s["idx"], s["case"]["h"], s["case"]["w"], s["attrs"], s["uv"], s["tex"])
            m.grads = dict(interp=s["g_attr"], sampled=s["g_tex"])
            meshes.append(m)
        b = MeshBatch(Rasterizer(), meshes)
        b.allocate_gradients()
        return dict(case=case, batch=b)
    return _pad_scene(case, seed)


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "render":
        from photara_drender_gb300.torch import render

        o = render(s["clip"], s["idx"], (c["h"], c["w"]), rasterizer=s["rasterizer"], vertex_attributes=s["attrs"],
                   vertex_uv=s["uv"], texture=s["tex"], cull_mode=c["cull"], address_mode=c["address"],
                   deferred_errors=c["deferred"])
        grads = torch.autograd.grad([o.interpolated, o.sampled], [s["clip"], s["attrs"], s["uv"], s["tex"]],
                                    [s["g_attr"], s["g_tex"]])
        return [o.raster, o.derivatives, o.interpolated, o.uv, o.sampled, *grads]
    if kind == "chain":
        from photara_drender_gb300.torch import interpolate, rasterize, texture

        r = s["rasterizer"]
        raster, deriv = rasterize(s["clip"], s["idx"], (c["h"], c["w"]), rasterizer=r, cull_mode=c["cull"])
        attr = interpolate(s["attrs"], raster, s["idx"], rasterizer=r)
        uv = interpolate(s["uv"], raster, s["idx"], rasterizer=r)
        sampled = texture(s["tex"], uv, raster, rasterizer=r, address_mode=c["address"])
        grads = torch.autograd.grad([attr, sampled], [s["clip"], s["attrs"], s["uv"], s["tex"]],
                                    [s["g_attr"], s["g_tex"]])
        return [raster, deriv, attr, uv, sampled, *grads]
    if kind == "bake":
        o = s["baker"].bake(s["pos"], s["nrm"], s["uv"], s["idx"], s["images"], s["mats"], s["eyes"],
                            visibility_masks=s["masks"], resolution=(c["atlas_h"], c["atlas_w"]), blend_mode=c["blend"],
                            visibility_mode=c["visibility"], pcf_radius=c["pcf"])
        return list(o[:5])
    if kind == "refine":
        o = s["baker"].refine_texture(s["init"], s["pos"], s["uv"], s["idx"], s["images"], s["mats"],
                                      visibility_masks=s["masks"], seam_uv_pairs=s["pairs"], steps=c["steps"],
                                      batch_size=c["batch"], seam_polish_steps=c["polish"],
                                      total_variation_weight=c["tv"], atlas_valid_mask=s["valid"], chart_ids=s["chart"])
        return list(o[:3])
    if kind == "batch":
        b = s["batch"]
        b.forward()
        b.backward()
        return [[m.outputs[k] for k in ("raster", "deriv", "interp", "uv", "sampled")]
                + [m.grads[k] for k in ("clip", "attributes", "uv_attributes", "texture")] for m in b.meshes]
    from photara_drender_gb300.padding import pad_texture_atlas

    return pad_texture_atlas(s["color"], s["valid"], c["margin"], coverage_mask=s["covered"], fill_unobserved=c["fill"],
                             maximum_fill_distance=c["distance"])


def _render_bytes(n, views, h, w, A, ch, th, tw):
    """Images out (raster, derivatives, attributes, uv, samples), upstream gradients in, mesh and texture in,
    their gradients out."""
    V, T = 6 * (n + 1) ** 2, 12 * n * n
    pixel = 16 + 16 + 4 * A + 8 + 4 * ch + 4 * A + 4 * ch
    return views * h * w * pixel + 2 * views * V * 16 + T * 12 + 2 * V * 4 * (A + 2) + 2 * th * tw * ch * 4


def work(case):
    c, kind = case, case["kind"]
    if kind in ("render", "chain"):
        ch = c.get("channels", 4)
        return dict(bytes=_render_bytes(c["n"], c["views"], c["h"], c["w"], c["attrs"], ch, c["tex_h"], c["tex_w"]),
                    flops=c["views"] * c["h"] * c["w"] * 200.0 + c["views"] * 12 * c["n"] ** 2 * 60.0)
    if kind == "batch":
        sizes = _batch_sizes(c)
        return dict(bytes=sum(_render_bytes(n, v, h, w, c["attrs"], 4, t, t) for n, v, h, w, t in sizes),
                    flops=sum(v * h * w * 250.0 + v * 12 * n * n * 60.0 for n, v, h, w, t in sizes))
    V, T = (6 * (c["n"] + 1) ** 2, 12 * c["n"] ** 2) if "n" in c else (0, 0)
    if kind == "bake":
        N = c["atlas_h"] * c["atlas_w"]
        photo = c["views"] * c["h"] * c["w"] * 4 * (c["channels"] + int(c["masks"]))
        return dict(bytes=N * 32 + photo + V * 32 + T * 12, flops=N * c["views"] * 60.0)
    if kind == "refine":
        N, P = c["atlas_h"] * c["atlas_w"], c["h"] * c["w"]
        polish = c["polish"] if c["pairs"] else 0
        # per step: texture and both moments read and written, the batch's uv, target and mask read
        return dict(bytes=(c["steps"] + polish) * N * 72.0 + c["steps"] * c["batch"] * P * 24.0 + c["views"] * P * 16.0,
                    flops=(c["steps"] + polish) * N * 3 * 15.0 + c["steps"] * c["batch"] * P * 60.0)
    N = c["atlas_h"] * c["atlas_w"]
    return dict(bytes=N * (8.0 * c["channels"] + 8), flops=N * 20.0)


# ---- float64 restatements -----------------------------------------------------------------------------

def _ids(clip, idx, h, w, cull="none"):
    """Winning triangle (id + 1, 0 for none) of every pixel of one view: nearest depth, ties to the lowest id."""
    p = clip.to(F64)[idx.long()]
    ok = (p[..., 3] > 1e-8).all(1)
    s = p[..., :2] / p[..., 3:].clamp_min(1e-8)
    d1, d2 = s[:, 1] - s[:, 0], s[:, 2] - s[:, 0]
    area = d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0]
    ok &= area.abs() > 1e-12
    if cull != "none":
        ok &= area > 0 if cull == "back" else area < 0
    size = torch.tensor([w, h], device=DEV, dtype=F64)
    lo = torch.floor((s.amin(1) * 0.5 + 0.5) * size).clamp_min(0)
    hi = torch.minimum(torch.ceil((s.amax(1) * 0.5 + 0.5) * size), size)
    ext = (hi - lo).clamp_min(0).long()
    cnt = torch.where(ok, ext[:, 0] * ext[:, 1], 0)
    tri = torch.nonzero(cnt)[:, 0]
    ends = cnt[tri].cumsum(0)
    best = torch.full((h * w,), 2.0, device=DEV, dtype=F64)
    found, a = [], 0
    cuts = torch.arange(1, int(cnt.sum()) // 4_000_000 + 2, device=DEV) * 4_000_000  # candidates of one go
    for b in [min(x + 1, len(tri)) for x in torch.searchsorted(ends, cuts).tolist()]:
        if b <= a:
            continue
        many = cnt[tri[a:b]]
        t = torch.repeat_interleave(tri[a:b], many)
        k = torch.arange(len(t), device=DEV) - torch.repeat_interleave(many.cumsum(0) - many, many)
        a = b
        px, py = lo[t, 0].long() + k % ext[t, 0], lo[t, 1].long() + k // ext[t, 0]
        at = torch.stack([(px + 0.5) * 2 / w - 1, (py + 0.5) * 2 / h - 1], -1)
        q = s[t] - at[:, None]
        e = torch.stack([q[:, i, 0] * q[:, j, 1] - q[:, i, 1] * q[:, j, 0] for i, j in ((1, 2), (2, 0), (0, 1))], -1)
        inside = (e * torch.sign(area[t])[:, None] >= -1e-7).all(1)
        t, at, pix = t[inside], at[inside], (py * w + px)[inside]
        z = _barycentric(p[t], at)[3]
        best.scatter_reduce_(0, pix, z, "amin")
        found.append((t, pix, z))
    ids = torch.full((h * w,), 1 << 40, device=DEV)
    for t, pix, z in found:
        win = z == best[pix]
        ids.scatter_reduce_(0, pix[win], t[win] + 1, "amin")
    return torch.where(ids == 1 << 40, 0, ids).reshape(h, w)


def _cross(a, b):
    return a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]


def _barycentric(p, at):
    """(b0, b1, area, depth) of corners p [N, 3, 4] at NDC samples at [N, 2]."""
    q = p[..., :2] - at[:, None] * p[..., 3:]
    a0, a1, a2 = _cross(q[:, 1], q[:, 2]), _cross(q[:, 2], q[:, 0]), _cross(q[:, 0], q[:, 1])
    A = a0 + a1 + a2
    z = (p[:, 0, 2] * a0 + p[:, 1, 2] * a1 + p[:, 2, 2] * a2) / (p[:, 0, 3] * a0 + p[:, 1, 3] * a1 + p[:, 2, 3] * a2)
    return a0 / A, a1 / A, A, z.clamp(-1, 1)


def _samples(ys, xs, h, w):
    return torch.stack([(xs + 0.5) * 2 / w - 1, (ys + 0.5) * 2 / h - 1], -1).to(F64)


def _wrap(i, n, mode):
    if mode == 0:
        return i.clamp(0, n - 1)
    if mode == 1:
        return i % n
    m = i % (2 * n)
    return torch.where(m < n, m, 2 * n - 1 - m)


def _taps(uv, h, w, mode=0):
    """Texel indices [N, 4] and weights [N, 4] of bilinear samples."""
    x, y = uv[:, 0] * w - 0.5, uv[:, 1] * h - 0.5
    bx, by = torch.floor(x.detach()), torch.floor(y.detach())
    fx, fy = x - bx, y - by
    x0, x1 = _wrap(bx.long(), w, mode), _wrap(bx.long() + 1, w, mode)
    y0, y1 = _wrap(by.long(), h, mode), _wrap(by.long() + 1, h, mode)
    return (torch.stack([y0 * w + x0, y0 * w + x1, y1 * w + x0, y1 * w + x1], -1),
            torch.stack([(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy], -1))


def _exact_render(s):
    """Images and gradients of rasterize -> interpolate, interpolate -> texture, view by view. None for the
    barycentric derivatives and the clip gradients: a few pixels on edge-on triangles, which one rounding of
    an edge test gives to a triangle or its neighbour, are larger than all others together."""
    c = s["case"]
    h, w, mode = c["h"], c["w"], ADDRESS[c.get("address", "clamp")]
    one = s["clip"].ndim == 2
    clips, g_attr, g_tex = (x[None] if one else x for x in (s["clip"], s["g_attr"], s["g_tex"]))
    attrs, uvs, idx = s["attrs"].to(F64).requires_grad_(True), s["uv"].to(F64).requires_grad_(True), s["idx"].long()
    tex = s["tex"].to(F64).reshape(-1, s["tex"].shape[2]).requires_grad_(True)
    total = [torch.zeros_like(x) for x in (attrs, uvs, tex)]
    images = []
    for k in range(clips.shape[0]):
        ids = _ids(clips[k].detach(), idx, h, w, c.get("cull", "none"))
        ys, xs = torch.nonzero(ids, as_tuple=True)
        tri = idx[ids[ys, xs] - 1]
        u, v, _, z = _barycentric(clips[k].detach().to(F64)[tri], _samples(ys, xs, h, w))
        u, v = u.clamp(0, 1), v.clamp(0, 1)
        bary = torch.stack([u, v, 1 - u - v], -1)[..., None]
        attr, uv = (attrs[tri] * bary).sum(1), (uvs[tri] * bary).sum(1)
        o, wt = _taps(uv, c["tex_h"], c["tex_w"], mode)
        smp = (tex[o] * wt[..., None]).sum(1)
        loss = (attr * g_attr[k][ys, xs]).sum() + (smp * g_tex[k][ys, xs]).sum()
        for t, r in zip(total, torch.autograd.grad(loss, [attrs, uvs, tex])):
            t += r
        row = []
        for val in (torch.stack([u, v, z, ids[ys, xs].to(F64)], -1), attr, uv, smp):
            im = torch.zeros((h, w, val.shape[-1]), device=DEV, dtype=F64)
            im[ys, xs] = val.detach()
            row.append(im)
        images.append(row)
    raster, attr, uv, smp = (images[0][j] if one else torch.stack([r[j] for r in images]) for j in range(4))
    return [raster, None, attr, uv, smp, None, total[0], total[1], total[2].reshape(s["tex"].shape)]


def _photo_views(s):
    """Per view: clip positions, the id image and the covered pixels' corners and barycentrics."""
    c = s["case"]
    clips = _clip(s["pos"], s["mats"])
    for k in range(c["views"]):
        ids = _ids(clips[k], s["idx"], c["h"], c["w"])
        ys, xs = torch.nonzero(ids, as_tuple=True)
        tri = s["idx"].long()[ids[ys, xs] - 1]
        b0, b1, _, z = _barycentric(clips[k].to(F64)[tri], _samples(ys, xs, c["h"], c["w"]))
        yield k, ids, ys, xs, tri, torch.stack([b0, b1, 1 - b0 - b1], -1)[..., None], z


def _exact_bake(s):
    """The shadow-map bake: color, confidence, valid and coverage masks (the source view is a whole number)."""
    c = s["case"]
    H, W = c["atlas_h"], c["atlas_w"]
    uv = s["uv"]
    flat = torch.cat([uv * 2 - 1, torch.zeros_like(uv[:, :1]), torch.ones_like(uv[:, :1])], 1)
    ids = _ids(flat, s["idx"], H, W)
    ty, tx = torch.nonzero(ids, as_tuple=True)
    tri = s["idx"].long()[ids[ty, tx] - 1]
    b0, b1, _, _ = _barycentric(flat.to(F64)[tri], _samples(ty, tx, H, W))
    bary = torch.stack([b0, b1, 1 - b0 - b1], -1)[..., None]
    pos, nrm = (s["pos"].to(F64)[tri] * bary).sum(1), (s["nrm"].to(F64)[tri] * bary).sum(1)
    nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    n = len(ty)
    acc, conf, top = torch.zeros((n, 3), device=DEV, dtype=F64), torch.zeros(n, device=DEV, dtype=F64), None
    for k, vid, ys, xs, _, _, z in _photo_views(s):
        h, w = c["h"], c["w"]
        depth = torch.full((h, w), float("nan"), device=DEV, dtype=F64)
        depth[ys, xs] = z
        M = torch.from_numpy(s["mats"][k]).to(DEV, F64)
        q = torch.cat([pos, torch.ones((n, 1), device=DEV, dtype=F64)], 1) @ M.T
        nd = q[:, :3] / q[:, 3:]
        ppx, ppy = (nd[:, 0] * 0.5 + 0.5) * w, (nd[:, 1] * 0.5 + 0.5) * h
        view = torch.from_numpy(s["eyes"][k]).to(DEV, F64) - pos
        dist = view.norm(dim=-1)
        cos = (nrm * view / dist[:, None]).sum(-1)
        ok = (q[:, 3] > 1e-8) & (nd.abs() <= 1).all(1) & (ppx < w) & (ppy < h) & (cos >= 0.05)
        seen, count = torch.zeros_like(cos), torch.zeros_like(cos)
        cx, cy, r = torch.floor(ppx).long(), torch.floor(ppy).long(), c["pcf"]
        for dy in range(-r, r + 1):
            for dx in range(-r, r + 1):
                X, Y = cx + dx, cy + dy
                inside = (X >= 0) & (Y >= 0) & (X < w) & (Y < h)
                dd = depth[Y.clamp(0, h - 1), X.clamp(0, w - 1)]
                inside &= ~torch.isnan(dd)
                count += inside
                seen += inside & (nd[:, 2] <= dd + 1e-3)
        vis = torch.where(count > 0, seen / count.clamp_min(1), 0.0) * ok
        o, wt = _taps(torch.stack([ppx / w, ppy / h], -1), h, w)
        if s["masks"] is not None:
            vis = vis * (s["masks"][k].to(F64).reshape(-1)[o] * wt).sum(1).clamp(0, 1)
        img = (s["images"][k].to(F64).reshape(h * w, -1)[o] * wt[..., None]).sum(1)
        alpha = img[:, 3] if img.shape[1] == 4 else 1.0
        if c["blend"] == "softmax":
            return None
        cf = vis * alpha * cos * ok
        if c["blend"] == "best_view":
            take = (cf > 0) & (cf >= conf)
            acc, conf = torch.where(take[:, None], img[:, :3], acc), torch.where(take, cf, conf)
        else:
            acc, conf = acc + img[:, :3] * cf[:, None], conf + cf
    div = conf if c["blend"] != "best_view" else torch.ones_like(conf)
    out = [torch.zeros((H, W, 4), device=DEV, dtype=F64)]
    out += [torch.zeros((H, W), device=DEV, dtype=F64) for _ in range(3)]
    out[0][ty, tx, :3] = torch.where(conf[:, None] > 0, acc / div.clamp_min(1e-300)[:, None], 0.0)
    out[0][ty, tx, 3] = (conf > 0).to(F64)
    out[1][ty, tx] = conf
    out[2][ty, tx] = (conf > 0).to(F64)
    out[3][ty, tx] = 1.0
    return [out[0], out[1], None, out[2], out[3]]


def _exact_refine(s):
    """The optimisation loop with the default options: color, loss history, seam loss history."""
    c = s["case"]
    H, W = c["atlas_h"], c["atlas_w"]
    cache, weights = [], []
    for k, _, ys, xs, tri, bary, _ in _photo_views(s):
        m = s["masks"][k][ys, xs].to(F64).clamp(0, 1)
        uv = (s["uv"].to(F64)[tri] * bary).sum(1)
        keep = m > 0
        o, wt = _taps(uv[keep], H, W)
        cache.append((o.int(), wt, s["images"][k][ys, xs][keep].to(F64), m[keep]))
        weights.append(float(m.sum()))
    x = s["init"].to(F64).reshape(-1, 3).clone()
    m1, m2 = torch.zeros_like(x), torch.zeros_like(x)
    hm = vm = None
    if c["tv"]:
        valid, chart = s["valid"] > 0.5, s["chart"]
        hm = (valid[:, 1:] & valid[:, :-1] & (chart[:, 1:] == chart[:, :-1]))[..., None]
        vm = (valid[1:] & valid[:-1] & (chart[1:] == chart[:-1]))[..., None]
        scale = c["tv"] / (max(int(hm.sum() + vm.sum()), 1) * 3)

    def adam(g, lr, t):
        m1.mul_(0.9).add_(g, alpha=0.1)
        m2.mul_(0.999).addcmul_(g, g, value=0.001)
        x.sub_(lr * (m1 / (1 - 0.9 ** t)) / ((m2 / (1 - 0.999 ** t)).sqrt_() + 1e-8)).clamp_(0, 1)

    hist, seam = [], []
    for step in range(c["steps"]):
        batch = [(step * c["batch"] + b) % c["views"] for b in range(c["batch"])]
        total = sum(weights[b] for b in batch)
        norm = 1.0 / (total * 3) if total > 0 else 0.0
        g, loss = torch.zeros_like(x), 0.0
        for b in batch:
            o, wt, target, m = cache[b]
            d = (x[o] * wt[..., None]).sum(1) - target
            robust = (d * d + 1e-6).sqrt()
            gg = d / robust * m[:, None] * norm
            loss = loss + (robust * m[:, None]).sum() * norm
            for j in range(4):
                g.index_add_(0, o[:, j], gg * wt[:, j:j + 1])
        if c["tv"]:
            X, G = x.reshape(H, W, 3), g.reshape(H, W, 3)
            for mask, a, b in ((hm, (slice(None), slice(None, -1)), (slice(None), slice(1, None))),
                               (vm, (slice(None, -1),), (slice(1, None),))):
                d = X[b] - X[a]
                t = d / (d * d + 1e-8).sqrt() * scale * mask
                G[b] += t
                G[a] -= t
        hist.append(loss)
        adam(g, 2.5e-4 + 0.5 * (5e-3 - 2.5e-4) * (1 + math.cos(math.pi * step / c["steps"])), step + 1)
    if c["pairs"]:
        m1.zero_()
        m2.zero_()
        pr = s["pairs"].to(F64)
        taps = [_taps(pr[:, j], H, W) for j in (0, 1)]
        for k in range(c["polish"]):
            d = (x[taps[0][0]] * taps[0][1][..., None]).sum(1) - (x[taps[1][0]] * taps[1][1][..., None]).sum(1)
            robust = (d * d + 1e-8).sqrt()
            seam.append(robust.sum() / (3 * len(pr)))
            gg, g = d / robust / (3 * len(pr)), torch.zeros_like(x)
            for sign, (o, wt) in zip((1.0, -1.0), taps):
                for j in range(4):
                    g.index_add_(0, o[:, j], sign * gg * wt[:, j:j + 1])
            adam(g, 1e-3, k + 1)
    empty = torch.zeros(0, device=DEV, dtype=F64)
    return [x.reshape(H, W, 3), torch.stack(hist), torch.stack(seam) if seam else empty]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("render", "chain"):
        return _exact_render(_render_scene(case, seed))
    if kind == "batch":
        return [_exact_render(s) for s in _batch_scenes(case, seed)]
    if kind == "bake" and case["visibility"] == "shadow_map":
        return _exact_bake(_photo_scene(case, seed))
    if kind == "refine":
        s = _photo_scene(case, seed)
        s["init"], s["chart"], s["valid"], s["pairs"] = _refine_extra(case, seed)
        return _exact_refine(s)
    return None  # ray visibility needs a ray tracer; padding copies colours
