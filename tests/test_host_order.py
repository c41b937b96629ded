"""The order of what the host code puts on its streams, on a CUDA runtime that
runs nothing (fake_cuda.py); no GPU."""
import re

import pytest

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


@pytest.mark.parametrize("kind", ["renderer", "side streams", "batch", "graph"])
@pytest.mark.parametrize("kernel", ["k_bin", "k_scan_tiles", "k_bricks", "k_gb_setup", "k_gb_big", "k_march"])
def test_counters_are_zero_after_a_failed_frame(tmp_path, kind, kernel):
    """A frame leaves the binning and raster counters zero by its last kernels.
    After one whose launches failed part of the way, the next frame clears them
    before its first kernel, once what was launched has run."""
    out = run(tmp_path, f"""
        kind, kernel = {kind!r}, {kernel!r}
        if kind in ("batch", "graph"):
            fake.fake_clear()
            b = R.Batch([(scene(), 32, 16, 32, 0)], use_graph=kind == "graph")
            b.shape = dict(b.shape, trace_per_scene=1)
            take("set-up")
            render = b.render
        else:
            fake.fake_clear()
            r, s, ids = loaded(overlap_raster=int(kind == "side streams"))
            take("set-up")
            render = lambda: frame(r, s, ids)
        fake.fake_fail(kernel.encode(), 0)
        out["failed"] = fails(render)
        take("bad")
        render()
        take("good")
        (b if kind in ("batch", "graph") else r).synchronize()
        fake.fake_clear()
        render()
        take("next")
    """)
    assert out["failed"]
    zeroed = lambda log: {tuple(x.split()[1:3]) for x in log if re.match(r"memset .* to 0 ", x)}  # noqa: E731
    first = lambda log, what: next(i for i, x in enumerate(log) if re.match(what, x))  # noqa: E731
    counters = {c for c in zeroed(out["set-up"]) if int(c[1]) in (4, 8, 4 * (32 // 8) ** 3)}
    assert {int(c[1]) for c in counters} == {4, 8, 256}
    good = out["good"]
    head = good[:first(good, "capture|launch|replay")]
    assert counters <= zeroed(head)
    assert not unfinished([x for x in out["bad"] if not x.endswith("FAILED")] + [x for x in head if "sync" in x])
    assert not counters & zeroed(out["next"])  # (and a good one needs no clearing)


@pytest.mark.parametrize("word,value", [("HEAVY_TOTAL", 5000), ("EXTRA_TOTAL", 100000)])
def test_graph_is_captured_again_after_the_slots_grew(tmp_path, word, value):
    """A captured frame holds the split bricks' arrays.  Once a frame's status
    made them larger, the freed ones must not be replayed."""
    out = run(tmp_path, f"""
        b = R.Batch([(scene(), 32, 16, 32, 0)], use_graph=True)
        status({word}, {value})
        b.render()
        status({word}, 0)
        fake.fake_clear()
        b.synchronize()
        take("grow")
        b.render()
        take("next")
        b.synchronize()
        fake.fake_clear()
        b.render()
        take("same")
    """)
    assert any(x.startswith("free") for x in out["grow"])
    assert any(x.startswith("capture") for x in out["next"])
    assert not any(x.startswith("capture") for x in out["same"])


def test_what_could_not_be_allocated_is_not_used(tmp_path):
    """A list that a frame needed larger and that no memory was found for is
    gone: the next frame's kernels get it with a capacity of 0, and it is
    allocated again once there is memory.  So are the maps of a new grid."""
    out = run(tmp_path, """
        r, s, ids = loaded()
        status(BIGTRI_TOTAL, 200000)
        frame(r, s, ids)
        fake.fake_fail(b"malloc", 0)
        out["failed"] = [fails(r.synchronize)]
        fake.fake_clear()
        status(BIGTRI_TOTAL, 0)
        frame(r, s, ids)
        take("without a list")
        r.synchronize()
        fake.fake_fail(b"malloc3d", 0)
        out["failed"].append(fails(r.set_grid_resolution, 64))
        fake.fake_fail(b"malloc3d", 0)
        out["failed"].append(fails(frame, r, s, ids))
        take("without maps")
        fake.fake_fail(b"", -1)
        frame(r, s, ids)
        take("with maps")
        out["grid"] = r.grid()[0]
    """)
    assert out["failed"] == [True, True, True]
    lists = [x.split()[1:] for x in out["without a list"] if x.startswith("records")]
    assert lists and all(cap == "0" for _, cap in lists)
    assert not any(x.startswith("launch") for x in out["without maps"])
    assert any(x.startswith("malloc3d") for x in out["with maps"]) and out["grid"] == 64


def test_a_kernel_has_one_shared_memory_limit(tmp_path):
    """The limit of a kernel's dynamic shared memory belongs to the process:
    were it set to what a call needs, a renderer on one thread could lower it
    between another's setting and launch.  So every call sets the same."""
    out = run(tmp_path, """
        rng = np.random.default_rng(0)
        rows = rng.random((1 << 15, 12), dtype=np.float32)
        r = R.Renderer(16, 16, grid_res=16)
        for log2 in (8, 13, 15, 17):
            r.mlp_init(R.mlp_desc(log2_table=log2))
            r.mlp_train_samples(rows, R.mlp_desc(log2_table=log2, steps=1))
            r.mlp_eval(rows[:100])
        take("train")
    """)["train"]
    limits, need = {}, {}
    for line in out:
        w = line.split()
        if w[0] == "attribute":
            limits.setdefault(w[1], set()).add(int(w[3]))
        if w[0] == "launch" and int(w[3]) > 48 << 10:
            need[w[1]] = max(need.get(w[1], 0), int(w[3]))
    assert any("encode_smem" in k for k in need)
    for k, n in need.items():
        assert len(limits[k]) == 1 and n <= min(limits[k]), (k, limits[k], n)
