"""Atlas padding by tiles, by bands, and by bands after the tiles gave up at any pass of either direction
(pdr_pad_texture_atlas_passes): colours, filled masks and statistics bit for bit the oracle's on every route."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import api
from photara_drender_gb300 import _native
from photara_drender_gb300.rasterizer import _ptr
from tests.gpu_util import same_bits
from tests.padding_cases import chart_atlas

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def pad(color, valid, cov, filled, margin, passes):
    h, w, ch = color.shape
    c, v, cv, f = (torch.tensor(x, device=DEV) for x in (color, valid, cov, filled))
    need = C.c_size_t()
    _native.call("pdr_pad_workspace_bytes", w, h, ch, C.byref(need))
    ws = torch.randint(0, 255, (need.value,), dtype=torch.uint8, device=DEV)
    stats = torch.empty(5, dtype=torch.int64, device=DEV)
    status = torch.zeros(_native.STATUS_WORDS, dtype=torch.int32, device=DEV)
    _native.call("pdr_pad_texture_atlas_passes", _ptr(c), ch, _ptr(v), _ptr(cv), _ptr(f), w, h, margin, 1, 0, 0.5, passes,
                 _ptr(ws), need.value, _ptr(stats), _ptr(status), C.c_void_p(torch.cuda.current_stream(DEV).cuda_stream))
    assert not status.any()
    return c.cpu().numpy(), f.cpu().numpy(), tuple(stats.tolist())


@pytest.mark.parametrize("h,w", [(1, 1), (1, 200), (300, 1), (31, 33), (32, 64), (33, 65), (64, 128), (97, 250), (290, 410)])
@pytest.mark.parametrize("sources", ["charts", "corner", "last corner", "column", "dots"])
def test_routes_agree_with_the_oracle(h, w, sources):
    rng = np.random.default_rng(h * 1000 + w)
    color, valid, cov, filled = chart_atlas(rng, h, w, 3 + (h + w) % 2)
    if sources != "charts":
        valid[:] = 0
        filled[:] = 0
        if sources == "corner":
            valid[0, 0] = 1
        elif sources == "last corner":
            valid[-1, -1] = 1
        elif sources == "column":
            valid[:, -1] = 1
        else:
            valid[rng.uniform(size=(h, w)) < 1e-3] = 1
        color = rng.uniform(size=color.shape).astype(np.float32)
        cov[:] = 1
    want_c, want_f, want = api.pad_texture_atlas(color, valid, 6, coverage_mask=cov, filled_mask=filled, fill_unobserved=True,
                                                 maximum_fill_distance=0, valid_threshold=0.5)
    for passes in (0, 1, 2, 3, 4, 6, 9, 14, 1 << 20):
        c, f, stats = pad(color, valid, cov, filled, 6, passes)
        assert stats == tuple(want), passes
        assert same_bits(c, want_c) and same_bits(f, want_f), passes
