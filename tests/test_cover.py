"""The brick kernels' coverage tests in their fast forms (csrc/vct_cover.h:
32- and 64-bit separating-axis columns, clamped 32-bit edge rows) decide every
voxel and sample as the plain 64/128-bit ones do.  Host build of the header
the kernels include; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fast_forms_match_the_plain_ones(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "cover_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wno-unknown-pragmas", "-I",
                    os.path.join(ROOT, "voxel_cone_tracing_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cover_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "60000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("0 differ")
