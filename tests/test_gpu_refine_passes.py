"""The refinement's passes at the edges of their tiles and shortcuts (csrc/refine.cu).

Adam: bit for bit the oracle's update over all magnitudes at which its quotients change form, and on texels without
gradient and moments. The fused TV + Adam pass: bit for bit the separate passes at ragged sizes. The photometric pass:
several pixels a thread, against the same taps summed in double precision."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import api
from photara_drender_gb300 import TextureBaker, _native
from photara_drender_gb300.baking import RefineOptionsC, RefineViewC
from photara_drender_gb300.rasterizer import _ptr
from tests.gpu_util import same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [1, 2, 40, 100000])
@pytest.mark.parametrize("betas,lr,eps", [((0.9, 0.999), 0.01, 1e-8), ((0.5, 0.25), 1e30, 1e-3)])
def test_adam_bits(step, betas, lr, eps):
    baker = TextureBaker(0)
    dev = baker.context.device
    rng = np.random.default_rng(step)
    n = 70001
    scale = 10.0 ** rng.uniform(-40, 18, (n, 3))
    tex = rng.uniform(-0.2, 1.2, (n, 3)).astype(np.float32)
    m = (rng.normal(size=(n, 3)) * scale).astype(np.float32)
    v = (rng.uniform(size=(n, 3)) * scale * np.where(rng.random((n, 1)) < 0.5, scale, 1.0)).astype(np.float32)
    g = (rng.normal(size=(n, 3)) * scale).astype(np.float32)
    g[rng.random(n) < 0.4] = 0.0
    m[rng.random(n) < 0.5] = 0.0
    v[rng.random(n) < 0.5] = 0.0
    still = rng.random(n) < 0.3
    m[still] = v[still] = g[still] = 0.0
    m[rng.random((n, 3)) < 0.05] = -0.0
    b1, b2 = betas
    bc1, bc2 = (float(np.float32(1) - np.float32(b) ** np.float32(step)) for b in betas)
    g4 = np.concatenate([g, np.zeros((n, 1), np.float32)], 1)
    d = [torch.tensor(x, device=dev) for x in (tex, g4, m, v)]
    _native.call("pdr_refine_adam", *(_ptr(t) for t in d), tex.size, lr, b1, b2, eps, bc1, bc2, 0.0, 1.0,
                 baker.context.stream())
    api.adam_update(tex, g, m, v, lr, b1, b2, eps, bc1, bc2, 0.0, 1.0)
    assert same_bits(d[0].cpu().numpy(), tex)
    assert same_bits(d[2].cpu().numpy(), m) and same_bits(d[3].cpu().numpy(), v)
    assert not d[1].any()


@pytest.mark.parametrize("shape", [(1, 1), (2, 31), (9, 32), (17, 33), (8, 256), (33, 257), (7, 600), (700, 3), (1500, 1030)])
@pytest.mark.parametrize("charts", [True, False])
def test_fused_tv_bits(shape, charts):
    baker = TextureBaker(0)
    dev, s = baker.context.device, baker.context.stream()
    h, w = shape
    rng = np.random.default_rng(h * 1000 + w)
    tex0 = rng.uniform(size=(h, w, 3)).astype(np.float32)
    tex0[rng.random((h, w)) < 0.2] = 0.5
    valid0 = (rng.random((h, w)) < 0.8).astype(np.uint8)
    valid = torch.tensor(valid0, device=dev)
    chart = torch.tensor(np.add.outer(np.arange(h) // 5 * 7, np.arange(w) // 11).astype(np.int32), device=dev)
    view = (RefineViewC * 1)()
    uv, target, mask = torch.zeros(2, device=dev), torch.zeros(3, device=dev), torch.zeros(1, device=dev)
    view[0].uv, view[0].target, view[0].mask, view[0].pixel_count = (uv.data_ptr(), target.data_ptr(), mask.data_ptr(), 1)
    vd = torch.frombuffer(bytearray(bytes(view)), dtype=torch.uint8).to(dev)
    weight = (C.c_double * 1)(1.0)
    o = RefineOptionsC(width=w, height=h, steps=3, batch_size=1, learning_rate=0.02, minimum_learning_rate=0.01,
                       photometric_epsilon=1e-3, adam_beta1=0.9, adam_beta2=0.999, adam_epsilon=1e-8, clamp_min=0.0,
                       clamp_max=1.0, seam_polish_steps=1, seam_learning_rate=1e-3, seam_epsilon=1e-4, tv_scale=1e-3,
                       tv_epsilon=1e-4)
    outs = []
    for fused in (False, True):
        tex, scratch = torch.tensor(tex0, device=dev), torch.full((h, w, 3), float("nan"), device=dev)
        grad = torch.full((h, w, 4), float("nan"), device=dev)
        m, v = torch.full_like(tex, float("nan")), torch.full_like(tex, float("nan"))
        loss = torch.empty(3, device=dev)
        o.texture_scratch = scratch.data_ptr() if fused else None
        _native.call("pdr_refine_run", C.byref(o), _ptr(vd), 1, C.cast(weight, C.c_void_p), 1, None, 0, _ptr(valid),
                     _ptr(chart) if charts else None, _ptr(tex), _ptr(grad), _ptr(m), _ptr(v), _ptr(loss), 0, s)
        outs.append([t.cpu().numpy() for t in (tex, m, v, grad)])
    for a, b in zip(*outs):
        assert same_bits(a, b)
    if h * w > 100:
        assert not same_bits(outs[1][0], tex0)


@pytest.mark.parametrize("pixels,batch", [((1,), 1), ((257, 1000, 3), 3), ((70000, 5, 69000, 30001), 4),
                                          ((400000, 260000, 1, 399999), 4)])
def test_photometric_rounds(pixels, batch):
    baker = TextureBaker(0)
    dev, s = baker.context.device, baker.context.stream()
    rng = np.random.default_rng(len(pixels) + pixels[0])
    tw, th, eps, norm = 61, 47, np.float32(0.1), np.float32(1e-3)
    tex = rng.uniform(size=(th * tw, 3)).astype(np.float32)
    views, keep = (RefineViewC * len(pixels))(), []
    # sums in double precision of each pixel's terms and of their magnitudes, from the shader's fp32 taps
    grad, size, count, loss = np.zeros((th * tw, 3)), np.zeros((th * tw, 3)), np.zeros(th * tw), 0.0
    for k, P in enumerate(pixels):
        uv = rng.uniform(-0.05, 1.05, (P, 2)).astype(np.float32)
        target = rng.uniform(size=(P, 3)).astype(np.float32)
        mask = (rng.uniform(size=P) * (rng.random(P) < 0.6)).astype(np.float32)
        t = [torch.tensor(x, device=dev) for x in (uv, target, mask)]
        keep.append(t)
        views[k].uv, views[k].target, views[k].mask = (x.data_ptr() for x in t)
        views[k].pixel_count = P
        xy = uv * np.array([tw, th], np.float32) - np.float32(0.5)
        base = np.floor(xy)
        f = (xy - base).astype(np.float64)
        base = base.astype(np.int64)
        taps = []
        for dy in (0, 1):
            for dx in (0, 1):
                o = np.clip(base[:, 1] + dy, 0, th - 1) * tw + np.clip(base[:, 0] + dx, 0, tw - 1)
                taps.append((o, np.abs(1 - dx - f[:, 0]) * np.abs(1 - dy - f[:, 1])))
        d = sum(tex[o].astype(np.float64) * w[:, None] for o, w in taps) - target
        robust = np.sqrt(d * d + float(eps) ** 2)
        m = mask.astype(np.float64)[:, None] * float(norm)
        loss += (robust * m).sum()
        for o, w in taps:
            for c in range(3):
                grad[:, c] += np.bincount(o, (d / robust * m)[:, c] * w, th * tw)
                size[:, c] += np.bincount(o, m[:, 0] * w, th * tw)
            count += np.bincount(o, minlength=th * tw)
    vd = torch.frombuffer(bytearray(bytes(views)), dtype=torch.uint8).to(dev)
    t_tex, out, t_loss = torch.tensor(tex, device=dev), torch.zeros((th * tw, 4), device=dev), torch.zeros(3, device=dev)
    _native.call("pdr_refine_photometric", _ptr(t_tex), tw, th, _ptr(vd), len(pixels), max(pixels), 0, batch, float(eps),
                 float(norm), _ptr(out), _ptr(t_loss), s)
    got = out.cpu().numpy().astype(np.float64)
    # a residual of values up to 1 is rounded by under 8 * 2^-24, divided by at least eps: 5e-6 of a term; then the
    # term's own roundings and the sum's, each at most 2^-24 of the terms' magnitudes
    bound = size * (5e-6 + (count[:, None] + 16) * 2.0 ** -24)
    assert (np.abs(got[:, :3] - grad) <= bound).all() and not got[:, 3].any()
    assert abs(t_loss[0].item() - loss) <= 1e-5 * loss and not t_loss[1:].any()


@pytest.mark.parametrize("pixels", [1, 255, 257, 70001])
@pytest.mark.parametrize("channels,external", [(3, True), (4, False)])
def test_prepare_view_in_one_pass(pixels, channels, external):
    """Target, mask, coordinates and weight of a view against the separate calls, bit for bit (the weight: sums of
    2^-10 steps, exact in any order), for coordinates at an address that is no multiple of 8."""
    baker = TextureBaker(0)
    dev, s = baker.context.device, baker.context.stream()
    rng = np.random.default_rng(pixels)
    V, T = 50, 30
    image = torch.tensor(rng.uniform(size=(pixels, channels)).astype(np.float32), device=dev)
    ext = torch.tensor((rng.integers(-200, 1400, pixels) / 1024).astype(np.float32), device=dev) if external else None
    raster = rng.uniform(size=(pixels, 4)).astype(np.float32)
    raster[:, 3] = rng.integers(0, T + 3, pixels)  # some ids past the last triangle
    raster = torch.tensor(raster, device=dev)
    idx = torch.tensor(rng.integers(0, V, (T, 3)).astype(np.int32), device=dev)
    uv = torch.rand(2 * V + 1, device=dev)[1:].view(V, 2)
    new = lambda *shape: torch.full(shape, 7.0, device=dev)  # noqa: E731
    t0, m0, u0 = new(pixels, 3), new(pixels), new(pixels, 2)
    t1, m1, u1 = new(pixels, 3), new(pixels), new(pixels, 2)
    weight = torch.zeros(64, dtype=torch.float64, device=dev)
    e = None if ext is None else _ptr(ext)
    _native.call("pdr_refine_prepare_view", _ptr(image), channels, e, _ptr(raster), pixels, _ptr(t0), _ptr(m0), s)
    _native.call("pdr_interpolate_forward", _ptr(uv), 0, V, 2, _ptr(idx), T, _ptr(raster), 1, pixels, _ptr(u0), s)
    _native.call("pdr_refine_prepare_view_uv", _ptr(image), channels, e, _ptr(raster), pixels, _ptr(uv), V, _ptr(idx), T,
                 _ptr(t1), _ptr(m1), _ptr(u1), _ptr(weight), s)
    for a, b in ((t0, t1), (m0, m1), (u0, u1)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert float(weight.sum()) == float(m0.double().sum())


@pytest.mark.parametrize("shape,steps,tv", [((256, 512), 120, False), ((256, 512), 120, True), ((32, 64), 160, True),
                                            ((1024, 512), 40, False)])
def test_overlapped_launches_read_final_values(shape, steps, tv):
    """Refinement steps launched while their predecessors run, against the same steps recorded in a graph, bit for bit.
    Every pixel samples one texel's centre (exact: sides are powers of two), and no two of a step the same one, so each
    gradient value is one term and zeros, whatever the order; its texels lie on lines that other CTAs have just written."""
    baker = TextureBaker(0)
    dev, s = baker.context.device, baker.context.stream()
    h, w = shape
    N = h * w
    rng = np.random.default_rng(h + steps)
    views, keep = (RefineViewC * 2)(), []
    for k in range(2):
        pick = rng.permutation(N)
        uv = np.stack([(pick % w + 0.5) / w, (pick // w + 0.5) / h], 1)
        t = [torch.tensor(x.astype(np.float32), device=dev) for x in (uv, rng.uniform(size=(N, 3)), rng.uniform(size=N))]
        keep.append(t)
        views[k].uv, views[k].target, views[k].mask = (x.data_ptr() for x in t)
        views[k].pixel_count = N
    vd = torch.frombuffer(bytearray(bytes(views)), dtype=torch.uint8).to(dev)
    valid = torch.tensor((rng.random((h, w)) < 0.8).astype(np.uint8), device=dev)
    weight = (C.c_double * 2)(N, N)
    o = RefineOptionsC(width=w, height=h, steps=steps, batch_size=1, learning_rate=0.02, minimum_learning_rate=0.01,
                       photometric_epsilon=1e-3, adam_beta1=0.9, adam_beta2=0.999, adam_epsilon=1e-8, clamp_min=0.0,
                       clamp_max=1.0, seam_polish_steps=0, seam_learning_rate=1e-3, seam_epsilon=1e-4,
                       tv_scale=1e-6 if tv else 0.0, tv_epsilon=1e-4)
    outs = []
    for mode in ("launches", "graph", "launches"):
        tex, scratch = torch.full((h, w, 3), 0.5, device=dev), torch.empty((h, w, 3), device=dev)
        grad, m, v = torch.empty((h, w, 4), device=dev), torch.empty_like(tex), torch.empty_like(tex)
        loss = torch.empty(steps, device=dev)
        o.texture_scratch = scratch.data_ptr() if tv else None
        args = (C.byref(o), _ptr(vd), 2, C.cast(weight, C.c_void_p), N, None, 0, _ptr(valid), None, _ptr(tex), _ptr(grad),
                _ptr(m), _ptr(v), _ptr(loss))
        if mode == "graph":
            g = C.c_void_p()
            _native.call("pdr_refine_graph_create", C.byref(g), *args, s)
            _native.call("pdr_refine_graph_launch", g, s)
            torch.cuda.synchronize()
            _native.call("pdr_refine_graph_destroy", g)
        else:
            _native.call("pdr_refine_run", *args, 1, s)
        outs.append([t.cpu().numpy() for t in (tex, m, v)])
    for other in outs[1:]:
        for a, b in zip(outs[0], other):
            assert same_bits(a, b)
