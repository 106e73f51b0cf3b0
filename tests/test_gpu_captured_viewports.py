"""A recorded render keeps reading its own viewport rows, however many others the rasterizer has seen since."""
import numpy as np
import pytest
import torch

import photara_drender_gb300 as pdr
from photara_drender_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("viewport", [(3.0, -2.0, 50.0, 61.5), [(0.0, 0.0, 64.0, 48.0), (10.0, 4.0, 30.0, 33.0)]])
def test_replay_after_many_other_viewports(viewport):
    dev = torch.device("cuda", 0)
    pos3, idx = S.icosphere(3)
    mats, _ = S.orbit_cameras(2)
    clip = torch.tensor(S.clip_positions(pos3, mats), device=dev)
    tidx = torch.tensor(idx.astype(np.int32), device=dev)
    attrs = torch.rand((pos3.shape[0], 3), device=dev)
    r = pdr.Rasterizer()

    def run():
        with torch.no_grad():
            o = pdr.render(clip, tidx, (48, 64), rasterizer=r, vertex_attributes=attrs, viewport=viewport,
                           deferred_errors=True)
        return o.raster, o.interpolated

    side = torch.cuda.Stream(dev)
    side.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(side):
        want = [t.clone() for t in run()]
    torch.cuda.current_stream(dev).wait_stream(side)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = run()
    for k in range(600):
        r.forward(clip[0], tidx, (2, 2 + k), output_barycentric_derivatives=False)
    torch.cuda.synchronize()
    # blocks of every small size, so that a freed row would be handed out again
    junk = [torch.full((n,), 5.0, device=dev) for n in (4, 8, 16, 64, 128) for _ in range(400)]
    for t in got:
        t.fill_(-1.0)
    g.replay()
    torch.cuda.synchronize()
    assert junk
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
