"""Single refinement steps directly behind the kernels that write their inputs, on one stream and without a wait: the
same values, bit for bit, as with a wait in between. Every pixel samples one texel's centre (exact: sides are powers of
two) and no two the same one, so sums do not depend on their order."""
import numpy as np
import pytest
import torch

from photara_drender_gb300 import TextureBaker, _native
from photara_drender_gb300.baking import RefineViewC
from photara_drender_gb300.rasterizer import _ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 32), (512, 1024)])
def test_single_steps_follow_their_inputs(shape):
    baker = TextureBaker(0)
    dev, s = baker.context.device, baker.context.stream()
    h, w = shape
    N = h * w
    rng = np.random.default_rng(h)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=dev)  # noqa: E731
    pick = rng.permutation(N)
    # a triangle per texel whose three corners are its centre
    uv = t(np.stack([(pick % w + 0.5) / w, (pick // w + 0.5) / h], 1))
    idx = torch.arange(N, dtype=torch.int32, device=dev)[:, None].expand(N, 3).contiguous()
    raster = torch.zeros((N, 4), device=dev)
    raster[:, 0], raster[:, 1] = 0.5, 0.25
    raster[:, 3] = torch.arange(1, N + 1, device=dev)
    image, ext = t(rng.uniform(size=(N, 3))), t(rng.uniform(0.1, 1, size=N))
    tex0 = t(rng.uniform(size=(N, 3)))
    pairs0 = torch.cat([uv, uv.flip(0)], 1)[: N // 2].contiguous()
    outs = []
    for wait in (True, False, False):
        sync = torch.cuda.synchronize if wait else (lambda: None)
        target, mask, coords = torch.zeros((N, 3), device=dev), torch.zeros(N, device=dev), torch.zeros((N, 2), device=dev)
        weight = torch.zeros(64, dtype=torch.float64, device=dev)
        view = (RefineViewC * 1)()
        view[0].uv, view[0].target, view[0].mask, view[0].pixel_count = (coords.data_ptr(), target.data_ptr(),
                                                                         mask.data_ptr(), N)
        table = torch.frombuffer(bytearray(bytes(view)), dtype=torch.uint8).to(dev)
        tex, grad, loss = torch.zeros((N, 3), device=dev), torch.zeros((N, 4), device=dev), torch.zeros(2, device=dev)
        m, v, pairs = torch.zeros((N, 3), device=dev), torch.zeros((N, 3), device=dev), torch.zeros((N // 2, 4), device=dev)
        torch.cuda.synchronize()
        tex.copy_(tex0)
        _native.call("pdr_refine_prepare_view_uv", _ptr(image), 3, _ptr(ext), _ptr(raster), N, _ptr(uv), N, _ptr(idx), N,
                     _ptr(target), _ptr(mask), _ptr(coords), _ptr(weight), s)
        sync()
        _native.call("pdr_refine_photometric", _ptr(tex), w, h, _ptr(table), 1, N, 0, 1, 1e-3, 1.0 / N, _ptr(grad),
                     _ptr(loss), s)
        sync()
        photometric = grad.clone()
        m.copy_(photometric[:, :3])
        v.copy_(m.square())
        sync()
        _native.call("pdr_refine_adam", _ptr(tex), _ptr(grad), _ptr(m), _ptr(v), N * 3, 0.01, 0.9, 0.999, 1e-8, 0.1, 0.01,
                     0.0, 1.0, s)
        sync()
        pairs.copy_(pairs0)
        sync()
        _native.call("pdr_refine_seam", _ptr(tex), w, h, _ptr(pairs), N // 2, 1e-4, 1.0 / N, _ptr(grad), _ptr(loss), 1, s)
        outs.append([x.cpu() for x in (photometric, tex, m, v, grad, mask, coords)])
        assert photometric.any() and grad.any()
    for other in outs[1:]:
        for a, b in zip(outs[0], other):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
