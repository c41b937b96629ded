"""The order of what the host code puts on its streams, on a CUDA runtime that
runs nothing (fake_cuda.py); no GPU."""
from tests.fake_cuda import run, unfinished


def test_setup_is_complete_when_a_call_returns(tmp_path):
    """The caller may change streams between any two calls, so the zeroing of
    the work arrays, which every frame expects to be zero, is complete when the
    call that allocates them returns: creation, a new grid, and a read-back
    after which the split bricks get more slots."""
    out = run(tmp_path, """
        r, s, ids = loaded()
        fake.fake_clear()
        r.set_grid_resolution(64)
        take("grid")
        R.Renderer(32, 16, grid_res=32)
        take("create")
        status(HEAVY_TOTAL, 5000)
        status(EXTRA_TOTAL, 100000)
        frame(r, s, ids)
        fake.fake_clear()
        r.read_frame()
        take("more slots")
        b = R.Batch([(scene(), 32, 16, 32, 0), (scene(), 16, 16, 64, 0)])
        take("batch")
        b.render()
        fake.fake_clear()
        b.synchronize()
        take("batch slots")
    """)
    for name, log in out.items():
        assert any(line.startswith("memset") for line in log), name
        assert not unfinished(log), (name, unfinished(log))
