"""Kernels launched programmatically (launch_next) start before their
predecessor is complete and wait in follows_previous().  What the predecessor
writes must not be read through __restrict__ pointers or __ldg: those promise
data that is constant for the kernel's whole life, and a compiler may move such
a load above the wait.  A check of the sources; no GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voxel_cone_tracing_gb300", "csrc")

# kernel or device function -> the pointers that a predecessor's writes reach
# it by (a helper's: of every kernel that calls it)
FED = {
    "k_scan.cu": {"k_scan_tiles": ["in"], "k_scan_add": ["in", "out", "tile_tot"]},
    "k_voxelize.cu": {
        "bin_one": ["count", "cursor"], "bin_tri": ["count", "cursor", "big", "big_count"],
        "k_bin": ["count", "cursor", "big", "big_count"], "k_bin_big": ["big", "big_count", "count", "cursor"],
        "brick_accumulate": ["list"], "brick_unit": ["offset", "list"], "k_bricks": ["offset", "list"],
        "k_bricks_linear": ["offset", "list"], "for_units": []},
    "k_raster.cu": {"warp_last_not_above": ["v"], "k_gb_big": [], "k_gb_resolve": []},
    "k_mipmap.cu": {"occ_raw_cell": [], "occ_pack_word": [], "occ_dilate_word": []},
    "vct_cone.cuh": {"direct_light": ["occlusion"]},
    "k_trace_frame.cu": {"shared_diffuse": ["far"], "k_shade": ["diffuse"]},
}
CONSTANT = r"__ldg\((in\.|vp|sp\.|w\.prefix|bw\.prefix|bb\.tri_prefix|r\.|m\.occ)"  # inputs of the whole frame


def functions(text):
    """(name, parameters, body) of the functions defined in a CUDA source."""
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in re.finditer(r"\b(\w+)\(([^;{}]*?)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(2), text[m.end():i]


@pytest.mark.parametrize("file", sorted(FED))
def test_no_constant_loads_of_a_predecessors_data(file):
    found = {}
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    for name, params, body in functions(text):
        if name in FED[file]:
            found[name] = params, body
    assert set(found) == set(FED[file])
    for name, (params, body) in found.items():
        for p in FED[file][name]:
            decl = [d for d in re.split(r",", params) if re.search(rf"\b{p}\s*$", d)]
            assert decl, (name, p)
            assert "__restrict__" not in decl[0], (name, p)
        for use in re.findall(r"__ldg\([^)]*", body):
            assert re.match(CONSTANT, use), (name, use)


def test_every_programmatic_kernel_is_listed():
    """Each kernel that waits for its predecessor stands in FED (the batch
    forms read through struct members, which promise nothing)."""
    for f in os.listdir(CSRC):
        if not f.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for name, params, body in functions(text):
            if name.startswith("k_") and re.search(r"follows_previous\(\)|for_units\(", body):
                known = name in FED.get(f, {}) or name in ("k_occupancy",) or "__restrict__" not in params
                assert known, (f, name)
