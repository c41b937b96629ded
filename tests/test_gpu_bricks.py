"""The brick kernels at the edges of their forms: triangles around 32 and 2048
voxels of extent (the 32-bit, 64-bit and 128-bit separating-axis tests),
columns and rows from one voxel to a whole brick, rounds of 1 to a few times
128 pairs, bricks that fall empty from frame to frame, and the allocation-free
path.  Contribution counts are integers: equal to the oracle's; level 0 within
1 LSB of its FP64 shading (the repository's bound for it)."""
import numpy as np
import pytest

from tests.helpers import tri_scene
from voxel_cone_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(n_grid, n, lo, hi, seed, spread=1.0):
    """n triangles of lo to hi voxels of extent around the grid's inside."""
    rng = np.random.default_rng(seed)
    v = 2.0 / n_grid
    at = rng.uniform(-0.9, 0.9, (n, 1, 3)) * spread
    size = rng.uniform(lo, hi, (n, 1, 3)) * v
    t = at + rng.uniform(-0.5, 0.5, (n, 3, 3)) * size
    t[::5, :, 1] = np.round(t[::5, :1, 1] / v) * v  # flat, on voxel faces
    mat = scenes.make_material((0.7, 0.5, 0.3), roughness=0.4)
    return tri_scene(np.clip(t, -60, 60), material=mat, lights=[((0.2, 0.5, 0.3),), ((-0.4, 0.1, 0.2),)])


def _voxels(vct, r, s):
    ids = vct.load_scene(r, s)
    vct.queue_scene(r, s, ids)
    r.render()
    return r.read_voxel_counts(), r.read_voxels(0)


@pytest.mark.parametrize("mode", [0, 1], ids=["raster", "conservative"])
@pytest.mark.parametrize("n_grid,n,lo,hi,spread", [
    (8, 1, 3, 9, 0.1), (8, 700, 0.1, 2, 1.0), (32, 129, 0.05, 0.6, 0.2), (32, 40, 20, 33, 1.0),
    (64, 30, 31, 34, 0.6), (64, 12, 100, 900, 0.5), (128, 150, 1900, 3900, 0.4), (64, 3000, 0.2, 12, 1.0)])
def test_counts_match_the_oracle(vct, oracle, mode, n_grid, n, lo, hi, spread):
    s = _scene(n_grid, n, lo, hi, n_grid + n, spread)
    want, cnt, _ = oracle.voxelize(s, oracle.Params(grid_res=n_grid, width=8, height=8, vox_mode=mode))
    r = vct.Renderer(8, 8, grid_res=n_grid, keep_counts=1, vox_mode=mode)
    got_cnt, got = _voxels(vct, r, s)
    r.close()
    assert cnt.sum() > 0
    np.testing.assert_array_equal(got_cnt, cnt)
    assert np.abs(got.astype(int) - want.astype(int)).max() <= 1


@pytest.mark.parametrize("cfg", [dict(), dict(vox_mode=1), dict(mip_mode=1), dict(storage=1, radiance_max=4.0)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()) or "default")
def test_bricks_that_fall_empty(vct, cfg):
    """Frames of different scenes through one renderer equal a new renderer's:
    bricks gain and lose their triangles, and none keeps old texels."""
    r = vct.Renderer(8, 8, grid_res=64, **cfg)
    first = True
    for seed, n, hi in ((1, 400, 20), (2, 9, 3), (3, 2000, 2), (4, 1, 1), (5, 300, 40)):
        s = _scene(64, n, 0.3, hi, seed, 0.3 * seed / 2)
        if first:
            ids = vct.load_scene(r, s)
        else:
            m = s.meshes[0]
            ids = [r.load_mesh(m.verts, m.indices, m.draw_objs)]
        first = False
        vct.queue_scene(r, s, ids)
        r.render()
        fresh = vct.Renderer(8, 8, grid_res=64, **cfg)
        fids = vct.load_scene(fresh, s)
        vct.queue_scene(fresh, s, fids)
        fresh.render()
        for level in (0, 1, 3):
            np.testing.assert_array_equal(r.read_voxels(level), fresh.read_voxels(level))
        fresh.close()
    r.close()


@pytest.mark.parametrize("mode", [0, 1], ids=["raster", "conservative"])
def test_lists_full_without_allocation(vct, mode):
    """5,000 large triangles at 64^3 through the path with fixed scratch (4,096
    large-triangle records, 256 split bricks of the 512): what does not fit is
    binned by its warp and run whole, and the texels are the renderer's."""
    import torch

    s = _scene(64, 5000, 25, 45, 77, 0.8)
    m = s.meshes[0]
    verts = torch.from_numpy(np.ascontiguousarray(m.verts, np.float32)).cuda()
    idx = torch.from_numpy(np.ascontiguousarray(m.indices, np.uint32).view(np.int32)).cuda()
    mat = torch.from_numpy(np.ascontiguousarray(m.tri_material(), np.uint32).view(np.int32)).cuda()
    mats = torch.from_numpy(np.frombuffer(np.ascontiguousarray(s.materials).tobytes(), np.uint8).copy()).cuda()
    d = vct.DeviceMesh()
    d.verts, d.indices, d.tri_material = verts.data_ptr(), idx.data_ptr(), mat.data_ptr()
    d.n_verts, d.n_tris = m.verts.shape[0], m.n_tris
    d.model[:] = [float(x) for x in np.asarray(s.models[0], np.float32)]
    r = vct.Renderer(8, 8, grid_res=64, vox_mode=mode)
    ids = vct.load_scene(r, s)
    vct.queue_scene(r, s, ids)
    r.render()
    want = r.read_voxels(0)
    r.close()
    out = torch.full((64, 64, 64, 4), 7, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        vct.voxelize_noalloc([d], mats.data_ptr(), s.materials.shape[0], s.lights, s.cube_size, 64, mode,
                             out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), want)
