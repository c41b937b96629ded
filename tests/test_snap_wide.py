"""Frames beyond 16,384 pixels a side: the raster's integer snapping is used
only where it equals FP64's and fits 32 bits (host build of the header, no
GPU), and wide frames show the oracle's triangles (GPU)."""
import os
import shutil
import subprocess

import pytest

from tests.test_gpu_raster import _check, _triangles

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_integer_snapping_stays_in_its_range(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "snap_wide_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "voxel_cone_tracing_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "snap_wide_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("0 of ")


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,n,lo,hi", [
    (16384, 3, 60, 1, 2000), (16385, 3, 60, 1, 2000), (3, 40000, 60, 1, 9000), (300000, 2, 80, 1, 200000),
    (600001, 1, 80, 1, 500000)])
def test_wide_frames_match_the_oracle(vct, oracle, w, h, n, lo, hi):
    """Visible triangles are integer results: equal, pixel for pixel."""
    t = _triangles(w, h, n, lo, hi, w + h)
    want = _check(vct, oracle, t, w, h)
    assert (want != 0xffffffff).any()
