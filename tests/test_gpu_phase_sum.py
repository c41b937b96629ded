"""The rendering phases, each switched on alone, add up to the whole frame: the
shader sums (specular + diffuse) + direct in FP32, products and sums apart, so
on opaque pixels the three frames' sum in that order is the frame bit for bit.
k_march plans other warps for every choice of phases; one that skipped or
misplaced a phase's would show."""
import numpy as np
import pytest

from voxel_cone_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu


def _frame(vct, s, w, h, phases, **cfg):
    r = vct.Renderer(w, h, keep_float_frame=1, grid_res=64, **cfg)
    ids = vct.load_scene(r, s)
    r.set_voxel_view_dir(7, 0.0)
    r.set_rendering_phases(*phases)
    vct.queue_scene(r, s, ids)
    r.render()
    f = r.read_frame(vct.FRAME_RGBA32F)[..., :3]
    r.close()
    return f


@pytest.mark.parametrize("cfg", [dict(), dict(far_share=0), dict(cone_set=1), dict(mip_mode=1), dict(full_march=1),
                                 dict(storage=1, radiance_max=4.0), dict(sampler=1)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()) or "default")
@pytest.mark.parametrize("lights", [1, 3])
def test_phases_sum_to_the_frame(vct, cfg, lights):
    w, h = 37, 23
    s = scenes.scene_sphere(seed=31, freq=12, width=w, height=h)
    s.materials["illum"] = 2
    s.lights = np.array([scenes.point_light(p, intensity=1.0) for p in
                         [(0.05, 0.35, 0.1), (-0.2, 0.4, -0.1), (0.1, 0.2, 0.3)][:lights]], scenes.LIGHT_DTYPE)
    whole, none, direct, unshadowed, diffuse, specular = (
        _frame(vct, s, w, h, ph, **cfg)
        for ph in [(1, 1, 1, 1), (0, 0, 0, 0), (1, 0, 0, 1), (1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0)])
    surface = (none == 0.0).all(-1)  # (elsewhere the clear colour)
    assert surface.sum() > w * h // 4
    np.testing.assert_array_equal(whole[surface], (specular + diffuse + direct)[surface])
    for f in (whole, direct, unshadowed, diffuse, specular):
        assert (f[surface] > 0.0).any()
        np.testing.assert_array_equal(f[~surface], none[~surface])
    # a shadow only takes light away (each light's term times at most 1 + 0.04)
    assert (unshadowed >= direct)[surface].all() and (unshadowed > direct)[surface].any()
