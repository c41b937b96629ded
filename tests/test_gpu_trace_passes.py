"""The frame tracer's passes (k_march, k_shade): scheduled shadow marches with
four-step and per-step empty-space tests, the alpha chains, lone pixels and
refracted cones, against the march that samples every step (full_march) of the
six maps (shadow_from_maps).  Skipped samples are exact zeros and the chains
hold the maps' own alphas, so the RGBA32F frames agree bit for bit."""
import numpy as np
import pytest

from voxel_cone_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(w, h, lights):
    s = scenes.scene_sphere(seed=31, freq=12, width=w, height=h)
    s.materials["illum"][::3] = 7
    s.materials["dissolve"][::3] = 0.5
    # inside the room, on the ceiling's plane, behind a wall, far outside the grid
    spots = [(0.05, 0.35, 0.1), (-0.2, 0.5, -0.1), (0.1, 0.2, -2.0), (400.0, 900.0, -50.0)]
    s.lights = np.array([scenes.point_light(p, intensity=1.0 + k) for k, p in enumerate(spots[:lights])],
                        scenes.LIGHT_DTYPE).reshape(-1)
    return s


def _frame(vct, s, w, h, **cfg):
    r = vct.Renderer(w, h, keep_float_frame=1, **cfg)
    ids = vct.load_scene(r, s)
    r.set_voxel_view_dir(7, 0.0)
    vct.queue_scene(r, s, ids)
    r.render()
    f = r.read_frame(vct.FRAME_RGBA32F)
    r.close()
    return f


@pytest.mark.parametrize("w,h,grid,lights,cfg", [
    (1, 1, 32, 1, dict()), (3, 2, 8, 1, dict()), (15, 17, 64, 0, dict()), (33, 31, 128, 4, dict()),
    (50, 37, 256, 2, dict(far_share=0)), (41, 20, 64, 3, dict(cone_set=1)), (41, 20, 64, 3, dict(mip_mode=1)),
    (47, 33, 64, 2, dict(storage=1, radiance_max=4.0)), (47, 33, 32, 2, dict(storage=1, mip_mode=2, cone_set=1)),
    (29, 18, 512, 1, dict()), (23, 9, 32, 4, dict(sampler=1)), (9, 5, 64, 0, dict(sampler=1, mip_mode=1, cone_set=1)),
    (13, 6, 32, 1, dict(sampler=1, storage=1))],
    ids=lambda v: "-".join(f"{k}{x}" for k, x in v.items()) or "default" if isinstance(v, dict) else str(v))
def test_passes_match_the_full_march(vct, w, h, grid, lights, cfg):
    s = _scene(w, h, lights)
    got = _frame(vct, s, w, h, grid_res=grid, **cfg)
    np.testing.assert_array_equal(got, _frame(vct, s, w, h, grid_res=grid, full_march=1, **cfg))
    np.testing.assert_array_equal(got, _frame(vct, s, w, h, grid_res=grid, shadow_from_maps=1, **cfg))
    assert np.isfinite(got).all()


@pytest.mark.parametrize("phases", [(1, 0, 0, 0), (1, 0, 0, 1), (0, 1, 0, 0), (0, 0, 1, 0), (0, 0, 0, 0)])
def test_phases_alone(vct, phases):
    """Each rendering phase switched on alone takes its own passes only: their
    sum over opaque pixels is the whole frame."""
    w, h = 37, 23
    s = scenes.scene_sphere(seed=31, freq=12, width=w, height=h)
    frames = []
    for ph in (phases, (1, 1, 1, 1)):
        r = vct.Renderer(w, h, keep_float_frame=1, grid_res=64)
        ids = vct.load_scene(r, s)
        r.set_voxel_view_dir(7, 0.0)
        r.set_rendering_phases(*ph)
        vct.queue_scene(r, s, ids)
        r.render()
        frames.append(r.read_frame(vct.FRAME_RGBA32F))
        r.close()
    assert np.isfinite(frames[0]).all()
    assert (frames[0][..., :3] <= frames[1][..., :3] + 1e-5).all() or phases == (1, 0, 0, 0)
    if not any(phases):
        g = frames[0][..., :3].reshape(-1, 3)
        assert set(map(tuple, np.unique(g, axis=0).round(4))) <= {(0.0, 0.0, 0.0), (0.15, 0.25, 0.25)}
