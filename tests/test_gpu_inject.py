"""Light injection's kernel (k_inject) at the edges of its shape: the smallest
grid (half a block of four-voxel groups), grids whose groups fill queues
exactly or leave them short, empty scenes and scenes where nearly every group
is occupied, no light and many.  Level 0 within 1 LSB of the FP64 oracle's
injection of the same attribute grids (the repository's bound for it)."""
import numpy as np
import pytest

from tests.helpers import tri_scene
from voxel_cone_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tris,size,lights", [
    (8, 1, 0.2, 1), (8, 60, 1.5, 2), (16, 3, 3.0, 0), (32, 400, 0.3, 10), (64, 900, 0.8, 3), (128, 5, 1.9, 1)])
def test_matches_the_oracle(vct, oracle, n, tris, size, lights):
    rng = np.random.default_rng(n + tris)
    t = rng.uniform(-0.9, 0.9, (tris, 1, 3)) + rng.uniform(-0.5, 0.5, (tris, 3, 3)) * size
    spots = [(tuple(rng.uniform(-0.8, 0.8, 3)), tuple(rng.uniform(0.2, 1, 3)), 1.0 + k) for k in range(lights)]
    s = tri_scene(t, material=scenes.make_material((0.7, 0.4, 0.2), emission=(0.1, 0.0, 0.3)), lights=spots)
    r = vct.Renderer(8, 8, grid_res=n)
    ids = vct.load_scene(r, s)
    r.set_light_injection(True)
    vct.queue_scene(r, s, ids)
    r.render()
    got = r.read_voxels(0)
    grids = r.read_injection_grids()
    r.close()
    want = oracle.inject(s, oracle.Params(grid_res=n, width=8, height=8), grids)
    assert (want[..., 3] > 0).any() or tris == 1  # (that one covers no sample: an empty grid)
    np.testing.assert_array_equal(got[..., 3], want[..., 3])
    assert np.abs(got.astype(int) - want.astype(int)).max() <= 1
