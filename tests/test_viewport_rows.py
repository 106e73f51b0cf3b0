"""The device rows of viewports that a rasterizer keeps (Rasterizer._device_viewports), with a context on the CPU: how
many are kept, which go first, that rows a CUDA graph capture has recorded never go, and the forms a viewport takes."""
import gc
import types
import weakref

import numpy as np
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


ROWS = [[0.0, 0.0, 9.0, 8.0], [1.0, 0.5, 7.0, 3.0], [2.0, -1.0, 4.0, 4.0]]


@pytest.mark.parametrize("form", [
    lambda v: v, lambda v: tuple(tuple(x) for x in v), lambda v: [None, *v[1:]], np.array, torch.tensor,
    lambda v: [np.array(x) for x in v], lambda v: [torch.tensor(x) for x in v], lambda v: iter(v),
    lambda v: [v[0], torch.tensor(v[1]), np.array(v[2])], lambda v: (tuple(x) for x in v)],
    ids=["lists", "tuples", "none", "array", "tensor", "arrays", "tensors", "iterator", "mixed", "generator"])
def test_forms_of_viewports_per_view(cpu_rasterizer, form):
    for _ in range(2):
        assert cpu_rasterizer._device_viewports(form(ROWS), 3, 9, 8).tolist() == ROWS


@pytest.mark.parametrize("form", [tuple, list, np.array, torch.tensor, lambda v: [np.float64(x) for x in v]],
                         ids=["tuple", "list", "array", "tensor", "scalars"])
def test_forms_of_one_viewport(cpu_rasterizer, form):
    for _ in range(2):
        assert cpu_rasterizer._device_viewports(form(ROWS[1]), 3, 9, 8).tolist() == [ROWS[1]] * 3


@pytest.mark.parametrize("bad", [(1.0, 2.0, 3.0), (0.0, 0.0, 0.0, 4.0), (0.0, 0.0, float("nan"), 4.0), [[0.0, 0.0, 1.0, 1.0]],
                                 torch.ones(2, 4), "abcd", ("a", "b", "c", "d")])
def test_what_is_no_viewport_is_refused(cpu_rasterizer, bad):
    with pytest.raises((ValueError, TypeError)):
        cpu_rasterizer._device_viewports(bad, 3, 9, 8)
    assert not cpu_rasterizer._viewport_cache
