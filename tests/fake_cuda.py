"""libvct.so's host code on the CUDA runtime of fake_cudart.cpp, in a child
process: no GPU, nothing runs, every stream-ordered call is logged."""
from __future__ import annotations

import json
import os
import re
import shutil
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "voxel_cone_tracing_gb300", "csrc")

PROLOGUE = """
import ctypes, json, sys
sys.path.insert(0, {root!r})
import numpy as np
fake = ctypes.CDLL({fake!r})
fake.fake_log.restype = ctypes.c_char_p
from voxel_cone_tracing_gb300 import renderer as R, scenes
log = lambda: fake.fake_log().decode().splitlines()
out = {{}}
def take(name):
    out[name] = log()
    fake.fake_clear()
def status(word, value):
    fake.fake_status({bytes}, word, value)
def fails(call, *a):
    try:
        call(*a)
    except R.VCTError:
        return True
    return False
def scene(w=32, h=16):
    return scenes.scene_sphere(seed=1, freq=4, width=w, height=h)
def loaded(**cfg):
    r, s = R.Renderer(32, 16, **dict(dict(grid_res=32), **cfg)), scene()
    r.set_voxel_view_dir(7, 0.0)
    return r, s, R.load_scene(r, s)
def frame(r, s, ids):
    R.queue_scene(r, s, ids)
    r.render()
"""


def status_words() -> list:
    """The names of FrameStatus's words, in order."""
    text = open(os.path.join(CSRC, "vct_internal.h")).read()
    body = re.search(r"struct FrameStatus \{(.*?)\n\};", text, re.S).group(1)
    return re.findall(r"^\s*(?:uint32_t|float) (\w+);", body, re.M)


def run(tmp_path, script: str) -> dict:
    """Runs `script` after PROLOGUE; returns what it left in `out`."""
    from voxel_cone_tracing_gb300 import build
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if cxx is None or not os.path.exists(nvcc):
        pytest.skip("needs g++ and the CUDA toolkit's headers")
    build.build()
    fake = str(tmp_path / "fake_cudart.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-I", inc, "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), "-o", fake], check=True)
    words = status_words()
    code = PROLOGUE.format(root=ROOT, fake=fake, bytes=4 * len(words)) + \
        "".join(f"{w.upper()} = {i}\n" for i, w in enumerate(words)) + textwrap.dedent(script) + "\nprint(json.dumps(out))"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT,
                       env=dict(os.environ, LD_PRELOAD=fake), timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return json.loads(r.stdout.splitlines()[-1])


def unfinished(log: list) -> list:
    """The log's stream-ordered work that no later synchronisation of its
    stream waits for."""
    left = []
    for line in log:
        m = re.match(r"(memset|copy|launch|replay) .*stream (\w+)$", line)
        if m:
            left.append((m.group(2), line))
        m = re.match(r"sync stream (\w+)$", line)
        if m:
            left = [x for x in left if x[0] != m.group(1)]
    return [x[1] for x in left]
