"""The batch forward through tile lists (pdr_render_batch_forward) for every tile configuration, with enough room for the
lists, with exactly enough and with too little (reported, and retried with what the report asks for): the images of the
visibility buffer (pdr_render_batch_direct), bit for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

import photara_drender_gb300 as pdr
from photara_drender_gb300 import _native
from photara_drender_gb300 import synthetic as S
from photara_drender_gb300.batch import CONFIGS, BatchConfigC, BatchMesh, MeshBatch
from photara_drender_gb300.rasterizer import _ptr

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def tile_lists(batch, config, capacity):
    cfg, segs, need = BatchConfigC(*config), C.c_uint64(), C.c_size_t()
    _native.call("pdr_render_batch_sizes", batch._table(), len(batch.meshes), C.byref(cfg), batch.A, C.byref(segs),
                 C.byref(need))
    offsets = torch.empty(segs.value + 1, dtype=torch.int32, device=DEV)
    lst = torch.full((max(capacity, 1) + 64,), -7, dtype=torch.int32, device=DEV)
    ws = torch.empty(need.value, dtype=torch.uint8, device=DEV)
    status = torch.zeros(_native.STATUS_WORDS, dtype=torch.int32, device=DEV)
    _native.call("pdr_render_batch_forward", batch._table(), len(batch.meshes), batch.A, batch.cull, batch.mode, C.byref(cfg),
                 _ptr(offsets), _ptr(lst), capacity, _ptr(ws), need.value, _ptr(status), batch.r.context.stream())
    st = status.tolist()
    assert (lst[capacity:] == -7).all() and not st[_native.STATUS_TILE_ENTRIES_HI]
    return st[_native.STATUS_TILE_ENTRIES], st[_native.STATUS_TILE_OVERFLOW]


@pytest.mark.parametrize("config", CONFIGS)
@pytest.mark.parametrize("attributes", [0, 3, 8])
@pytest.mark.parametrize("cull", ["none", "back"])
def test_tile_lists_give_the_direct_images(config, attributes, cull):
    rng = np.random.default_rng(attributes)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=DEV)  # noqa: E731
    meshes = []
    for sub, views, h, w, textured in ((2, 2, 48, 64, True), (3, 3, 97, 90, True), (0, 1, 130, 17, False)):
        pos3, idx = S.icosphere(sub)
        mats, _ = S.orbit_cameras(views, aspect=w / h)
        meshes.append(BatchMesh(
            clip=t(S.clip_positions(pos3, mats)), indices=torch.tensor(idx.astype(np.int32), device=DEV), height=h, width=w,
            attributes=t(rng.uniform(size=(pos3.shape[0], attributes))) if attributes else None,
            uv_attributes=t(S.spherical_uv(pos3)) if textured else None,
            texture=t(rng.uniform(size=(20, 30, 4))) if textured else None))
    batch = MeshBatch(pdr.Rasterizer(0), meshes, cull_mode=cull, address_mode="mirror")
    batch.forward()
    want = [{k: v.clone() for k, v in m.outputs.items()} for m in meshes]

    def images_agree():
        for m, w in zip(meshes, want):
            for k, v in w.items():
                assert torch.equal(m.outputs[k].view(torch.int32), v.view(torch.int32)), k
                m.outputs[k].fill_(-3.0)

    entries, overflow = tile_lists(batch, config, 100000)
    assert entries > 0 and not overflow
    images_agree()
    again, overflow = tile_lists(batch, config, entries // 3)
    assert again == entries and overflow
    assert tile_lists(batch, config, again) == (entries, 0)
    images_agree()
