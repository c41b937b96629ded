"""The G-buffer raster (k_gb_setup, k_gb_big) at its edges: pixel boxes around
the 64 pixels a setup thread rasters itself, around the 32x32-pixel tiles of
the larger ones, clipped and screen-filling triangles, frames smaller than a
tile, and more large triangles than the record list first holds.  Visible
triangles are integer results: equal to the oracle's, pixel for pixel."""
import math

import numpy as np
import pytest

from tests.helpers import tri_scene
from voxel_cone_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu


def _triangles(w, h, n, lo, hi, seed):
    """n triangles whose pixel boxes measure lo to hi pixels a side, anywhere
    on (and a little beyond) a w x h frame, at depths 1 to 3."""
    rng = np.random.default_rng(seed)
    centre = rng.uniform(-0.1, 1.1, (n, 1, 2)) * (w, h)
    size = rng.uniform(lo, hi, (n, 1, 2))
    corner = rng.uniform(-0.5, 0.5, (n, 3, 2))
    corner = (corner - corner.min(1, keepdims=True)) / np.ptp(corner, axis=1, keepdims=True) - 0.5
    # a quarter on whole pixel centres: samples on edges and corners
    px = centre + corner * size
    px[::4] = np.floor(px[::4]) + 0.5
    z = rng.uniform(1.0, 3.0, (n, 3, 1))
    tan = math.tan(math.radians(30.0))
    ndc = px / (w, h) * 2.0 - 1.0
    return np.concatenate([ndc * z * (tan * w / h, tan), -z], 2)


def _check(vct, oracle, tris, w, h):
    s = tri_scene([[tuple(map(float, v)) for v in t] for t in tris], cube_size=4.0, view=scenes.mat_identity(),
                  proj=scenes.perspective(math.radians(60.0), w / h, 0.01, 10.0))
    want = oracle.gbuffer(s, oracle.Params(grid_res=8, width=w, height=h))["tri_id"]
    r = vct.Renderer(w, h, grid_res=8)
    ids = vct.load_scene(r, s)
    for _ in range(2):
        vct.queue_scene(r, s, ids)
        r.render()
        np.testing.assert_array_equal(r.read_gbuffer()["tri_id"], want)
    r.close()
    return want


@pytest.mark.parametrize("w,h,n,lo,hi", [
    (1, 1, 5, 1, 40), (31, 5, 20, 1, 12), (33, 65, 40, 6, 10), (160, 90, 400, 0.2, 9), (97, 64, 60, 7, 9),
    (160, 90, 200, 30, 34), (257, 131, 100, 60, 140), (320, 200, 300, 1, 700), (64, 2000, 30, 1, 1500)])
def test_boxes(vct, oracle, w, h, n, lo, hi):
    want = _check(vct, oracle, _triangles(w, h, n, lo, hi, w + h + n), w, h)
    assert (want != 0xffffffff).any()


def test_clipped(vct, oracle):
    """Across the near plane and the guard band, through and behind the eye."""
    rng = np.random.default_rng(5)
    t = rng.uniform(-1.0, 1.0, (150, 3, 3)) * (3.0, 3.0, 2.0)
    t[::3] *= (40.0, 40.0, 1.0)
    want = _check(vct, oracle, t, 203, 77)
    assert (want != 0xffffffff).any()


def test_more_records_than_the_list_holds(vct, oracle):
    """70,000 large triangles on a list of 65,536: it grows, the frame is
    drawn again, and the ones past its end appear."""
    t = _triangles(200, 120, 70000, 10, 14, 9)
    t[:, :, :] *= np.linspace(3.0, 1.0, len(t))[:, None, None]  # later ones nearer
    want = _check(vct, oracle, t, 200, 120)
    assert (want[want != 0xffffffff] >= 65536).any()
