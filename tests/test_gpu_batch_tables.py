"""A batch call's tables belong to the call: a recorded forward and adjoint of a MeshBatch replays after the host memory
of the call is gone and reused, and batches whose tables take several pieces equal their meshes rendered alone. The
adjoint's workspace may start at any multiple of 8 bytes."""
import ctypes as C
import gc

import numpy as np
import pytest
import torch

import photara_drender_gb300 as pdr
from photara_drender_gb300 import _native
from photara_drender_gb300 import synthetic as S
from photara_drender_gb300.batch import BatchMesh, MeshBatch
from photara_drender_gb300.rasterizer import _ptr

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def mesh(rng, sub, views, h, w):
    pos3, idx = S.icosphere(sub)
    mats, _ = S.orbit_cameras(views, aspect=w / h)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=DEV)  # noqa: E731
    m = BatchMesh(clip=t(S.clip_positions(pos3, mats)), indices=torch.tensor(idx.astype(np.int32), device=DEV), height=h,
                  width=w, attributes=t(rng.uniform(size=(pos3.shape[0], 2))))
    m.grads["interp"] = t(rng.normal(size=(views, h, w, 2)))
    return m


def check(r, meshes):
    for m in meshes:
        one = BatchMesh(clip=m.clip, indices=m.indices, height=m.height, width=m.width, attributes=m.attributes)
        one.grads["interp"] = m.grads["interp"]
        single = MeshBatch(r, [one])
        single.forward()
        single.backward()
        for k in ("raster", "deriv", "interp"):
            assert torch.equal(m.outputs[k].view(torch.int32), one.outputs[k].view(torch.int32)), k
        for k in ("clip", "attributes"):  # sums of the same terms in another order
            d, top = float((m.grads[k] - one.grads[k]).abs().max()), float(one.grads[k].abs().max())
            assert d <= 1e-4 * top + 1e-7, (k, d, top)


@pytest.mark.parametrize("views", [1, 60, 150])
def test_tables_in_pieces(views):
    rng = np.random.default_rng(views)
    meshes = [mesh(rng, 2, views, 20, 24), mesh(rng, 1, 3, 33, 17)]
    r = pdr.Rasterizer(0)
    b = MeshBatch(r, meshes)
    b.forward()
    b.backward()
    check(r, meshes)


def test_recorded_batch_replays_with_its_own_tables():
    rng = np.random.default_rng(1)
    meshes = [mesh(rng, 2, 3, 40, 56), mesh(rng, 3, 2, 64, 48)]
    r = pdr.Rasterizer(0)
    b = MeshBatch(r, meshes)
    b.allocate_gradients()
    side = torch.cuda.Stream(DEV)
    side.wait_stream(torch.cuda.current_stream(DEV))
    with torch.cuda.stream(side):
        b.forward()
        b.backward()
    torch.cuda.current_stream(DEV).wait_stream(side)
    torch.cuda.synchronize(DEV)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        b.forward()
        b.backward()
    # what the calls allocated on the host is free: use it for something else
    gc.collect()
    junk = [np.full(n, 0xA5, np.uint8) for n in range(512, 65536, 512) for _ in range(8)]
    for m in meshes:  # other positions; the outputs have to follow them
        m.clip[..., :2] *= 0.9
        for t in (*m.outputs.values(), m.grads["clip"], m.grads["attributes"]):
            t.fill_(-1.0)
    g.replay()
    torch.cuda.synchronize(DEV)
    assert junk
    check(r, meshes)


def test_adjoint_workspace_at_a_multiple_of_8():
    rng = np.random.default_rng(2)
    meshes = [mesh(rng, 2, 2, 31, 29), mesh(rng, 1, 1, 16, 16)]
    r = pdr.Rasterizer(0)
    b = MeshBatch(r, meshes)
    b.forward()
    b.allocate_gradients()
    ws = torch.empty(b.workspace.numel() + 8, dtype=torch.uint8, device=DEV)
    _native.call("pdr_render_batch_backward", b._table(), len(meshes), b.A, b.mode, C.byref(b.config), _ptr(ws[8:]),
                 b.workspace.numel(), _ptr(b.status), r.context.stream())
    check(r, meshes)
