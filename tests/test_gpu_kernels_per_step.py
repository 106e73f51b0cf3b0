"""RenderFwdBwd.kernels_per_step against the kernel nodes of one step recorded into a CUDA graph."""
import ctypes as C

import numpy as np
import pytest
import torch

import photara_drender_gb300 as pdr
from photara_drender_gb300 import synthetic as S
from photara_drender_gb300.pipeline import RenderFwdBwd

pytestmark = pytest.mark.gpu


# a small texture; one larger than L2 that the views sample densely enough to sort their tiles, and one that they do not;
# two groups of views, of which the second has a view too few to sort
CASES = [(3, 96, (64, 48, 4)), (4, 1024, (2048, 4096, 4)), (3, 96, (2048, 4096, 4))]


@pytest.mark.parametrize("views,side,texture,kind", [(*c, k) for c in CASES for k in ("direct", "tile lists", "unfused")]
                         + [(17, 2048, (2048, 4096, 4), "direct")])
def test_count_matches_a_recorded_step(views, side, texture, kind):
    pos3, idx = S.icosphere(2)
    mats, _ = S.orbit_cameras(views)
    dev = torch.device("cuda", 0)
    clip = torch.tensor(S.clip_positions(pos3, mats), device=dev)
    V = pos3.shape[0]
    tidx = torch.tensor(idx.astype(np.int32), device=dev)
    attrs, uv = torch.rand((V, 1), device=dev), torch.tensor(S.spherical_uv(pos3).astype(np.float32), device=dev)
    tex, ga = torch.rand(texture, device=dev), torch.rand((views, side, side, 1), device=dev)
    gs = torch.rand((views, side, side, 4), device=dev)
    pipe = RenderFwdBwd(pdr.Rasterizer(), tidx, V, views, side, side, 1, texture, fused=kind != "unfused",
                        direct=kind == "direct")
    pipe.step(clip, attrs, uv, tex, ga, gs)
    torch.cuda.synchronize()
    cu, stream = C.CDLL("libcuda.so.1"), torch.cuda.Stream(dev)
    handle, graph, n = C.c_void_p(stream.cuda_stream), C.c_void_p(), C.c_size_t()
    assert cu.cuStreamBeginCapture_v2(handle, 2) == 0  # CU_STREAM_CAPTURE_MODE_RELAXED
    pipe.step(clip, attrs, uv, tex, ga, gs, stream=handle)
    assert cu.cuStreamEndCapture(handle, C.byref(graph)) == 0
    assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0
    kinds = []
    for node in nodes:
        k = C.c_int(-1)
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(k)) == 0
        kinds.append(k.value)
    assert cu.cuGraphDestroy(graph) == 0
    assert kinds.count(0) == pipe.kernels_per_step()  # CU_GRAPH_NODE_TYPE_KERNEL
