"""Uneven multi-mesh batches in one launch (no counterpart in the reference, which renders one mesh per
call): many meshes, each with its own views, resolution and texture, run through one visibility pass, one
shading launch and one adjoint launch (include/pdr_capi.h pdr_render_batch_direct, pdr_render_batch_backward).
The tile configurations are those of pdr_render_batch_forward, the tile-list forward with the same outputs;
nothing of the passes here depends on them.
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass, field
from typing import Dict, List, Optional, Sequence, Tuple

import torch

from . import _native
from .rasterizer import Rasterizer, _ptr, _viewports

CONFIGS: Tuple[Tuple[int, int, int], ...] = ((16, 8, 128), (16, 16, 128), (16, 16, 256))
_MODES = {"none": 0, "back": 1, "front": 2}
_ADDRESS = {"clamp": 0, "wrap": 1, "mirror": 2}


class RenderMeshC(C.Structure):
    """include/pdr_capi.h pdr_render_mesh."""
    _fields_ = [
        ("clip_positions", C.c_void_p), ("indices", C.c_void_p), ("viewports", C.c_void_p),
        ("attributes", C.c_void_p), ("uv_attributes", C.c_void_p), ("texture", C.c_void_p),
        ("views", C.c_uint32), ("vertex_count", C.c_uint32), ("triangle_count", C.c_uint32), ("width", C.c_uint32),
        ("height", C.c_uint32), ("texture_width", C.c_uint32), ("texture_height", C.c_uint32),
        ("raster", C.c_void_p), ("barycentric_derivatives", C.c_void_p), ("interpolated", C.c_void_p),
        ("uv", C.c_void_p), ("sampled", C.c_void_p), ("grad_interpolated", C.c_void_p),
        ("grad_sampled", C.c_void_p), ("grad_clip_positions", C.c_void_p), ("grad_attributes", C.c_void_p),
        ("grad_uv_attributes", C.c_void_p), ("grad_texture", C.c_void_p),
    ]


class BatchConfigC(C.Structure):
    _fields_ = [("tile_width", C.c_uint32), ("tile_height", C.c_uint32), ("stage_triangles", C.c_uint32)]


@dataclass
class BatchMesh:
    """One mesh of a batch: inputs (device tensors) and the output / gradient buffers the batch fills."""
    clip: torch.Tensor                      # [views, V, 4]
    indices: torch.Tensor                   # [T, 3] int32
    height: int
    width: int
    attributes: Optional[torch.Tensor] = None   # [V, A]
    uv_attributes: Optional[torch.Tensor] = None  # [V, 2]
    texture: Optional[torch.Tensor] = None  # [th, tw, 4]
    viewports: Optional[torch.Tensor] = None  # [views, 4]
    outputs: Dict[str, torch.Tensor] = field(default_factory=dict)
    grads: Dict[str, torch.Tensor] = field(default_factory=dict)


class MeshBatch:
    """A fixed set of meshes rendered forward and backward together."""

    def __init__(self, rasterizer: Rasterizer, meshes: Sequence[BatchMesh], cull_mode: str = "none",
                 address_mode: str = "clamp", config: Tuple[int, int, int] = (16, 16, 256)):
        self.r = rasterizer
        dev = rasterizer.context.device
        self.meshes = list(meshes)
        if not self.meshes:
            raise ValueError("a batch needs at least one mesh")
        A = {m.attributes.shape[1] if m.attributes is not None else 0 for m in self.meshes}
        if len(A) != 1:
            raise ValueError("all meshes of a batch share one attribute count")
        self.A = A.pop()
        self.cull, self.mode = _MODES[cull_mode], _ADDRESS[address_mode]
        f = dict(dtype=torch.float32, device=dev)
        for m in self.meshes:
            views = m.clip.shape[0]
            m.indices = m.indices.to(dev, torch.int32).contiguous()
            if m.viewports is None:
                m.viewports, _ = _viewports(None, views, m.width, m.height, dev)
            shape = (views, m.height, m.width)
            # outputs already attached to the mesh (e.g. by another batch holding it) are reused
            need = {"raster": 4, "deriv": 4}
            if m.attributes is not None:
                need["interp"] = self.A
            if m.uv_attributes is not None:
                need["uv"] = 2
            if m.texture is not None:
                need["sampled"] = 4
            for name, channels in need.items():
                if name not in m.outputs:
                    m.outputs[name] = torch.empty(shape + (channels,), **f)
        self.status = torch.zeros(_native.STATUS_WORDS, dtype=torch.int32, device=dev)
        self.set_config(config)

    # -- native structures -------------------------------------------------------------------------------
    def _table(self):
        arr = (RenderMeshC * len(self.meshes))()
        for k, m in enumerate(self.meshes):
            c = arr[k]
            c.clip_positions, c.indices, c.viewports = m.clip.data_ptr(), m.indices.data_ptr(), m.viewports.data_ptr()
            c.views, c.vertex_count, c.triangle_count = m.clip.shape[0], m.clip.shape[1], m.indices.shape[0]
            c.width, c.height = m.width, m.height
            if m.attributes is not None:
                c.attributes, c.interpolated = m.attributes.data_ptr(), m.outputs["interp"].data_ptr()
            if m.uv_attributes is not None:
                c.uv_attributes, c.uv = m.uv_attributes.data_ptr(), m.outputs["uv"].data_ptr()
            if m.texture is not None:
                c.texture, c.sampled = m.texture.data_ptr(), m.outputs["sampled"].data_ptr()
                c.texture_height, c.texture_width = m.texture.shape[0], m.texture.shape[1]
            c.raster, c.barycentric_derivatives = m.outputs["raster"].data_ptr(), m.outputs["deriv"].data_ptr()
            g = m.grads
            for name, attr in (("interp", "grad_interpolated"), ("sampled", "grad_sampled"),
                               ("clip", "grad_clip_positions"), ("attributes", "grad_attributes"),
                               ("uv_attributes", "grad_uv_attributes"), ("texture", "grad_texture")):
                if name in g:
                    setattr(c, attr, g[name].data_ptr())
        return arr

    def set_config(self, config: Tuple[int, int, int]) -> None:
        """The tile configuration of pdr_render_batch_forward; the passes here do not depend on it."""
        if tuple(config) not in CONFIGS:
            raise ValueError(f"batch configuration must be one of {CONFIGS}")
        self.config = BatchConfigC(*config)
        segs, ws, direct = C.c_uint64(), C.c_size_t(), C.c_size_t()
        _native.call("pdr_render_batch_sizes", self._table(), len(self.meshes), C.byref(self.config), self.A,
                     C.byref(segs), C.byref(ws))
        _native.call("pdr_render_batch_direct_workspace_bytes", self._table(), len(self.meshes), self.A, C.byref(direct))
        self.segments = segs.value
        self.workspace = torch.empty(max(ws.value, direct.value, 1), dtype=torch.uint8, device=self.r.context.device)

    # -- passes --------------------------------------------------------------------------------------------
    def forward(self, stream=None) -> None:
        """Renders every view of every mesh."""
        s = stream if stream is not None else self.r.context.stream()
        _native.call("pdr_render_batch_direct", self._table(), len(self.meshes), self.A, self.cull, self.mode,
                     _ptr(self.workspace), self.workspace.numel(), s)

    def allocate_gradients(self) -> None:
        for m in self.meshes:
            f = dict(dtype=torch.float32, device=m.clip.device)
            for name, src in (("clip", m.clip), ("attributes", m.attributes), ("uv_attributes", m.uv_attributes),
                              ("texture", m.texture)):
                if src is not None and name not in m.grads:
                    m.grads[name] = torch.empty(src.shape, **f)

    def backward(self, stream=None) -> None:
        """Adjoints of the last forward; upstream gradients are m.grads['interp'] / m.grads['sampled']."""
        ctx = self.r.context
        s = stream if stream is not None else ctx.stream()
        self.allocate_gradients()
        self.status.zero_()
        _native.call("pdr_render_batch_backward", self._table(), len(self.meshes), self.A, self.mode,
                     C.byref(self.config), _ptr(self.workspace), self.workspace.numel(), _ptr(self.status), s)

    def autotune(self, configs: Sequence[Tuple[int, int, int]] = CONFIGS, reps: int = 3,
                 backward: bool = True) -> Dict[Tuple[int, int, int], float]:
        """Times forward (+ backward) of this batch. Neither depends on the tile configuration (that of
        pdr_render_batch_forward), so they are timed once and every configuration gets that time; the first is
        kept. Returns {config: median milliseconds}."""
        dev = self.r.context.device
        for cfg in configs:
            self.set_config(cfg)
        samples = []
        for timed in range(reps + 1):  # the first untimed
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize(dev)
            e0.record()
            self.forward()
            if backward:
                self.backward()
            e1.record()
            torch.cuda.synchronize(dev)
            if timed:
                samples.append(e0.elapsed_time(e1))
        times = {tuple(cfg): sorted(samples)[len(samples) // 2] for cfg in configs}
        self.set_config(min(times, key=times.get))
        return times
