"""The raster's vertex snapping in integer arithmetic (csrc/vct_snap.h
snap_scaled) equals the FP64 rounding of (g + 1) * 128 * extent wherever it
decides.  Host build of the header the kernels include; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_snap_scaled_matches_fp64_rounding(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "snap_scaled_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "voxel_cone_tracing_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "snap_scaled_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("0 of ")
    left, spread = (int(x) for x in r.stdout.split(", ")[1].split(" left")[0].split(" of "))
    assert left < spread // 20
