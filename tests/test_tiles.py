"""The tiles of the G-buffer raster's large triangles (csrc/vct_tiles.h): their
count beside the records', and the origins of those that a full record list's
last box does not have.  Host build of the header the kernels include; no
GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tiles_lie_in_their_box(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "tiles_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", "-I",
                    os.path.join(ROOT, "voxel_cone_tracing_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "tiles_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("0 faults")
