"""Meshes of a batch whose gradient buffers are the same or overlap receive the sum of what each alone adds (one mesh at
two resolutions sharing its parameters, say); the other meshes' buffers are as always. Against every mesh's adjoint alone, summed
in double precision on the host; the tolerance is the sums' order, as for the batch against its meshes."""
import numpy as np
import pytest
import torch

import photara_drender_gb300 as pdr
from photara_drender_gb300 import synthetic as S
from photara_drender_gb300.batch import BatchMesh, MeshBatch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)
NAMES = ("clip", "attributes", "uv_attributes", "texture")


def make(rng, sub, views, h, w, attrs, textured=True):
    pos3, idx = S.icosphere(sub)
    mats, _ = S.orbit_cameras(views, aspect=w / h)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=DEV)  # noqa: E731
    m = BatchMesh(clip=t(S.clip_positions(pos3, mats)), indices=torch.tensor(idx.astype(np.int32), device=DEV), height=h,
                  width=w, attributes=t(rng.uniform(size=(pos3.shape[0], attrs))) if attrs else None,
                  uv_attributes=t(S.spherical_uv(pos3)) if textured else None,
                  texture=t(rng.uniform(size=(16, 24, 4))) if textured else None)
    if attrs:
        m.grads["interp"] = t(rng.normal(size=(views, h, w, attrs)))
    if textured:
        m.grads["sampled"] = t(rng.normal(size=(views, h, w, 4)))
    return m


def alone(r, m):
    one = BatchMesh(clip=m.clip, indices=m.indices, height=m.height, width=m.width, attributes=m.attributes,
                    uv_attributes=m.uv_attributes, texture=m.texture)
    one.grads.update({k: m.grads[k] for k in ("interp", "sampled") if k in m.grads})
    b = MeshBatch(r, [one])
    b.forward()
    b.backward()
    return {k: one.grads[k].cpu().numpy().astype(np.float64).ravel() for k in NAMES if k in one.grads}


# (which meshes' buffer of a name starts where in one buffer, in floats): equal starts share it, close ones overlap
@pytest.mark.parametrize("attrs,shared", [
    (3, {k: {0: 0, 2: 0} for k in NAMES}),
    (3, {"attributes": {0: 0, 1: 40, 2: 8}, "clip": {1: 0, 2: 0}}),
    (8, {"uv_attributes": {0: 0, 1: 2}}),
    (0, {"clip": {0: 0, 1: 4, 2: 128}, "texture": {1: 0, 2: 0}}),
    (1, {})])
def test_sums_into_shared_buffers(attrs, shared):
    rng = np.random.default_rng(attrs + len(shared))
    r = pdr.Rasterizer(0)
    meshes = [make(rng, 2, 2, 40, 33, attrs), make(rng, 1, 3, 24, 24, attrs), make(rng, 2, 2, 65, 80, attrs)]
    parts = [alone(r, m) for m in meshes]
    want, got = {}, {}
    for name in NAMES:
        starts = shared.get(name, {})
        size = max([starts[k] + parts[k][name].size for k in starts], default=0)
        buffer, total = torch.full((size,), float("nan"), device=DEV), np.zeros(size)
        for k, m in enumerate(meshes):
            if name not in parts[k]:
                continue
            source = {"clip": m.clip, "attributes": m.attributes, "uv_attributes": m.uv_attributes, "texture": m.texture}[name]
            if k in starts:
                n = parts[k][name].size
                m.grads[name] = buffer[starts[k]:starts[k] + n].view(source.shape)
                total[starts[k]:starts[k] + n] += parts[k][name]
            else:
                m.grads[name] = torch.full(source.shape, float("nan"), device=DEV)
                want[name, k], got[name, k] = parts[k][name], m.grads[name]
        if starts:
            want[name, "shared"], got[name, "shared"] = total, buffer
    b = MeshBatch(r, meshes)
    for _ in range(2):  # overwritten, not accumulated, from call to call
        b.forward()
        b.backward()
    for key, w in want.items():
        g = got[key].cpu().numpy().astype(np.float64).ravel()
        assert np.abs(g - w).max() <= 1e-4 * np.abs(w).max() + 1e-7, key
