"""The device rows of viewports that a rasterizer keeps (Rasterizer._device_viewports), with a context on the CPU: how
many are kept, which go first, and that rows a CUDA graph capture has recorded never go."""
import gc
import types
import weakref

import pytest
import torch

from photara_drender_gb300 import rasterizer as R


@pytest.fixture
def cpu_rasterizer(monkeypatch):
    monkeypatch.setattr(R, "Context", lambda *a, **k: types.SimpleNamespace(device=torch.device("cpu")))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: None)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda *a: None)
    capturing = [False]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    r = R.Rasterizer(0)
    r.capturing = capturing
    return r


def others(r, n, start=1):
    for k in range(start, start + n):
        r._device_viewports(None, 1, 1000 + k, 7)


def test_captured_rows_are_never_dropped(cpu_rasterizer):
    r = cpu_rasterizer
    single, several = (1.0, 2.0, 30.0, 40.0), [(0.0, 0.0, 9.0, 8.0), (1.0, 0.0, 9.0, 8.0)]
    r._device_viewports(single, 3, 64, 48)  # made before the capture, where the upload is allowed
    r._device_viewports(several, 2, 64, 48)
    r.capturing[0] = True
    kept = [weakref.ref(r._device_viewports(single, 3, 64, 48)), weakref.ref(r._device_viewports(several, 2, 64, 48))]
    r.capturing[0] = False
    others(r, 3 * R._VIEWPORT_CACHE)
    gc.collect()
    assert [k() is not None for k in kept] == [True, True]
    assert kept[0]().tolist() == [list(single)] * 3 and kept[1]().tolist() == [list(v) for v in several]
    assert len(r._viewport_cache) == R._VIEWPORT_CACHE


def test_least_recently_used_rows_go_first(cpu_rasterizer):
    r = cpu_rasterizer
    first, second = (weakref.ref(r._device_viewports(None, 1, w, 5)) for w in (11, 12))
    for k in range(4):
        others(r, R._VIEWPORT_CACHE // 2, start=1000 * k)
        assert r._device_viewports(None, 1, 11, 5) is first()
    assert first() is not None and second() is None
