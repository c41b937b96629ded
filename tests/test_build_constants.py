"""The constants that a build may override (-DVCT_...) tune launches; none of
them fixes a layout that several kernels and buffers agree on."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voxel_cone_tracing_gb300", "csrc")

TUNING = {
    "VCT_BRICK_THREADS", "VCT_BRICK_ROUND",  # static_asserts bound them
    "VCT_MARCH_MIN_BLOCKS", "VCT_MARCH_WARPS", "VCT_SHADE_MIN_BLOCKS", "VCT_TRACE_BATCH_MIN_BLOCKS",
    "VCT_TRACE_BATCH_SHARE_MIN_BLOCKS", "VCT_MIP_TMA_MIN_BLOCKS",  # residency
    "VCT_SHADOW_UNROLL", "VCT_FIRST_UNROLL", "VCT_TRACE_PIPE", "VCT_FAR_SHORT_TAIL", "VCT_LOD_FTZ",
    "VCT_SKIP_EMPTY_RGBA", "VCT_SKIP_MAX_LOD", "VCT_HEAVY_SPLIT", "VCT_FUSE_BRICK_MIPS"}  # forms of one result


def test_overridable_constants_fix_no_layout():
    """A sharing group is 4x2 pixels of an 8x4-pixel warp in the groups' far
    fields, in k_march's lanes and in k_shade's: one value for all."""
    found = set()
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h", ".cpp")):
            found |= set(re.findall(r"#ifndef (VCT_\w+)\n#define", open(os.path.join(CSRC, f)).read()))
    assert found <= TUNING
