"""The raster kernels' division by a viewport size without a division (csrc/ndc_axis.cuh NdcAxis) rounds
exactly like the division: tests/native/ndc_axis_check.cpp, compiled for the host."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotient_by_reciprocal_rounds_like_the_division(tmp_path):
    exe = str(tmp_path / "ndc_axis_check")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O2", "-ffp-contract=off",
                    os.path.join(HERE, "native", "ndc_axis_check.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
