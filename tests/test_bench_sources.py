"""The source files whose hash says whether bench.py's recorded DRAM bytes belong to the current code are those that the
timed stages' kernels are compiled from: each stage's launching file and all it includes (of csrc; the C header holds no
device code), and for the adjoint the file that launches the order of its tiles."""
import os
import re

import pytest

import bench

CSRC = os.path.join(os.path.dirname(os.path.abspath(bench.__file__)), "photara_drender_gb300", "csrc")


def included(name, seen=None):
    seen = set() if seen is None else seen
    if name not in seen:
        seen.add(name)
        with open(os.path.join(CSRC, name)) as f:
            for other in re.findall(r'^#include "(\w[\w.]*)"', f.read(), re.M):
                included(other, seen)
    return seen


@pytest.mark.parametrize("stage,launches,also", [("visibility+shade", "visibility.cu", set()),
                                                 ("render_backward", "fused.cu", {"visibility.cu"})])
def test_recorded_sources(stage, launches, also):
    assert set(bench.KERNEL_SOURCES[stage]) == included(launches) | also
    assert len(bench.KERNEL_SOURCES[stage]) == len(set(bench.KERNEL_SOURCES[stage]))
