"""What the engine's speed is measured on: the calls a program makes through
``voxel_cone_tracing_gb300.renderer``, over the sizes they come in.

``listed()`` names the cases, ``draw()`` gives more of the same ranges,
``prepare()`` builds what a program holds before the call (a renderer with
its scene loaded and one frame behind it), ``run()`` is one pass through the
public entry points, ``work()`` what a pass cannot do without, and ``exact()``
the learned term's values in 64 bits.

Scenes are the repository's own kind: the box room with a noise-displaced
sphere and cuboids in it, seeded materials, point lights and a camera that
differs a little from seed to seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from voxel_cone_tracing_gb300 import renderer as R
from voxel_cone_tracing_gb300 import scenes as S

FRAME = {"kind": "frame", "width": 1920, "height": 1080, "grid": 256, "tris": 499_290, "cones": 9, "mips": "aniso",
         "coverage": "raster2x", "hdr": False, "far_share": 1, "overlap": 0, "lights": 1, "glass": False,
         "sampler": "texture", "inject": False, "learned": False, "read": "device"}


def _frame(name, **kw):
    return dict(FRAME, name=name, **kw)


def listed():
    return [
        # The smallest call: a thumbnail of the plain method (64^3 grid, isotropic mips, six 60-degree
        # cones, room + 2 cuboids), read back to the host each time: latency and launches count.
        _frame("thumbnail", width=256, height=256, grid=64, tris=34, cones=6, mips="iso", read="host"),
        # The reference's default grid (128^3) at 720p: an interactive viewer's frame.
        _frame("viewer_720p", width=1280, height=720, grid=128, tris=72_010),
        # The repository's headline frame: 1080p, 256^3, half a million triangles.
        _frame("headline_1080p"),
        # The same frame by the reference's own rule, every pixel marching all of its cones.
        _frame("per_pixel_1080p", far_share=0),
        # A window of no round size, exact coverage, three lights, a glass material, raster beside voxelize.
        _frame("window_1367x771", width=1367, height=771, grid=128, tris=120_011, coverage="sat", lights=3, glass=True,
               overlap=1),
        # The precision workload: half-float maps at 512^3, radiance up to 16, two million triangles.
        _frame("hdr_512", grid=512, tris=1_997_514, coverage="sat", hdr=True),
        # Static geometry, light injected every frame from the attribute grids.
        _frame("injected_1080p", inject=True),
        # The learned diffuse term in place of the diffuse cones (the judge checks 1/256 of the pixels).
        _frame("learned_1080p", learned=True),
        # The FP32 software sampler, the accuracy mode, on a small frame.
        _frame("software_sampler", width=320, height=180, grid=64, tris=5_010, sampler="software"),
        # A render farm's step: scenes of uneven size per frame, captured in a graph, frames read back.
        {"name": "batch_16", "kind": "batch", "scenes": 16, "layout": 16, "min_tris": 1_000, "max_tris": 400_000,
         "max_grid": 256},
        # The voxelizer alone into a caller's tensor.
        {"name": "voxelize_128", "kind": "voxelize", "grid": 128, "tris": 200_010, "coverage": "raster2x", "lights": 2},
        # The learned term trained on from a checkpoint's parameters on explicit rows, as after a change of light.
        {"name": "train", "kind": "train", "rows": 1 << 18, "batch": 1 << 18, "steps": 12, "log2_table": 15},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["per_pixel", "hdr", "inject", "learned", "software", "batch", "voxelize", "train"])
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(3, 16), "layout": rng.randint(0, 9999), "min_tris": 1_000,
                "max_tris": _log(rng, 20_000, 400_000), "max_grid": rng.choice([128, 256])}
    if kind == "voxelize":
        return {"kind": "voxelize", "grid": rng.choice([32, 64, 128, 256]), "tris": _log(rng, 1_000, 400_000),
                "coverage": rng.choice(["raster2x", "sat"]), "lights": rng.randint(0, 4)}
    if kind == "train":
        rows = _log(rng, 1 << 14, 1 << 18)
        return {"kind": "train", "rows": rows, "batch": rng.choice([rows, max(1000, rows // 3)]),
                "steps": rng.randint(4, 12), "log2_table": rng.choice([13, 14, 15])}
    c = dict(FRAME, width=_log(rng, 200, 1920), grid=rng.choice([64, 128, 256]), tris=_log(rng, 1_000, 499_000),
             cones=rng.choice([9, 9, 6]), mips=rng.choice(["aniso", "aniso", "aniso", "iso", "both"]),
             coverage=rng.choice(["raster2x", "sat"]), overlap=rng.randint(0, 1), lights=rng.choice([1, 1, 2, 3]),
             glass=rng.random() < 0.3, read=rng.choice(["device", "device", "host"]))
    c["height"] = max(120, min(1080, int(c["width"] * rng.uniform(0.5, 0.8))))
    if kind == "per_pixel":
        c["far_share"] = 0
    elif kind == "hdr":
        c.update(hdr=True, grid=rng.choice([128, 256, 512]), tris=_log(rng, 30_000, 1_500_000), glass=False,
                 mips=rng.choice(["aniso", "aniso", "iso"]))
    elif kind == "inject":
        c["inject"] = True
    elif kind == "learned":
        c.update(learned=True, mips="aniso")
    elif kind == "software":
        c.update(sampler="software", width=_log(rng, 120, 320), grid=rng.choice([32, 64]), tris=_log(rng, 1_000, 20_000),
                 lights=1)
        c["height"] = max(80, int(c["width"] * 9 / 16))
    return c


# ------------------------------------------------------------------ scenes ----
@functools.lru_cache(maxsize=8)
def _sphere_grid(n):
    """Six n x n faces of a cube blown up to the unit sphere: points, triangles."""
    t = np.tan((np.arange(n + 1) / n * 2 - 1) * (math.pi / 4))
    a, b = np.meshgrid(t, t, indexing="ij")
    one = np.ones_like(a)
    faces = [(one, a, b), (-one, b, a), (b, one, a), (a, -one, b), (a, b, one), (b, a, -one)]
    p = np.stack([np.stack(f, -1) for f in faces])
    p /= np.linalg.norm(p, axis=-1, keepdims=True)
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None]).reshape(-1)
    quad = np.concatenate([np.stack([i, i + n + 1, i + n + 2], 1), np.stack([i, i + n + 2, i + 1], 1)])
    tris = np.concatenate([quad + f * (n + 1) * (n + 1) for f in range(6)]).astype(np.uint32)
    return p, tris


def _blob(rng, n_tris, mats, amplitude=0.05):
    """A displaced sphere of about n_tris triangles, one draw object per face; smooth normals from the
    displaced surface's own tangents."""
    n = max(2, int(round(math.sqrt(n_tris / 12.0))))
    p, tris = _sphere_grid(n)
    dirs = rng.normal(size=(8, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    freqs, phase, amps = rng.uniform(2, 9, 8), rng.uniform(0, 2 * math.pi, 8), rng.uniform(0.5, 1.0, 8)
    wave = freqs * (p @ dirs.T) + phase
    noise = (amps * np.sin(wave)).sum(-1) / amps.sum()
    slope = ((amps * freqs * np.cos(wave))[..., None] * dirs).sum(-2) / amps.sum()
    pos = p * (1 + amplitude * noise)[..., None]
    nrm = p - amplitude * (slope - (slope * p).sum(-1, keepdims=True) * p)
    nrm /= np.linalg.norm(nrm, axis=-1, keepdims=True)
    verts = np.zeros((p.shape[0] * p.shape[1] * p.shape[2], 8), np.float32)
    verts[:, :3], verts[:, 3:6] = pos.reshape(-1, 3), nrm.reshape(-1, 3)
    per = 6 * n * n
    runs = np.array([(per * f, per, mats[f % len(mats)]) for f in range(6)], S.DRAWOBJ_DTYPE)
    return S.Mesh(verts, tris, runs)


def _scene(rng, width, height, tris, lights=1, hdr=False, glass=False):
    mats = [S.default_material()]

    def mat(**kw):
        mats.append(S.make_material(rng.uniform(0.1, 0.9, 3), roughness=rng.uniform(0.1, 1.0), **kw))
        return len(mats) - 1

    meshes, models = [S.box_room([mat() for _ in range(5)])], [S.mat_identity()]
    n_blobs = 4 if hdr else (1 if tris > 200 else 0)
    for _ in range(n_blobs):
        ids = [mat(illum=7, dissolve=0.6) if glass and f == 0 else mat() for f in range(6)]
        meshes.append(_blob(rng, max(48, (tris - 10) // n_blobs), ids))
        lo, hi = ((0.08, 0.16) if hdr else (0.2, 0.28))
        models.append(S.trs(translate=rng.uniform([-0.2, -0.3, -0.25], [0.2, -0.1, 0.0]),
                            scale=np.full(3, rng.uniform(lo, hi))))
    for _ in range(32 if hdr else 2):
        glow = hdr and rng.uniform() < 0.3
        ids = [mat(emission=rng.uniform(0, 20, 3)) if glow else mat() for _ in range(6)]
        meshes.append(S.cuboid(ids))
        models.append(S.trs(translate=rng.uniform([-0.42, -0.45, -0.45], [0.42, 0.1, 0.1]), rot=S.random_rotation(rng),
                            scale=rng.uniform(0.03, 0.15, 3)))
    lt = np.array([S.point_light(rng.uniform([-0.3, 0.3, -0.2], [0.3, 0.45, 0.2]), intensity=12.0 if hdr else 1.0)
                   for _ in range(lights)], S.LIGHT_DTYPE).reshape(-1)
    eye = np.array([0.0, 0.02, 0.49]) + rng.uniform(-0.03, 0.0, 3)
    view = S.look_at(eye, (rng.uniform(-0.05, 0.05), -0.08, -0.5))
    proj = S.perspective(math.radians(60.0), width / height, 0.01, 10.0)
    return S.Scene(meshes, models, np.array(mats, S.MATERIAL_DTYPE), lt, view, proj, S.ROOM_CUBE_SIZE)


class _DeviceFrame:
    """The renderer's RGBA8 frame as a CUDA array; keeps the renderer alive."""

    def __init__(self, r):
        self.renderer = r
        self.__cuda_array_interface__ = {"shape": (r.height, r.width, 4), "typestr": "|u1", "strides": None,
                                         "data": (r.frame_device_ptr(), False), "version": 3}


# ----------------------------------------------------------------- prepare ----
def prepare(case, seed):
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 77])
    return {"frame": _prepare_frame, "batch": _prepare_batch, "voxelize": _prepare_voxelize,
            "train": _prepare_train}[case["kind"]](case, seed, rng)


def _network(rng, log2_table, n_levels=16):
    table = rng.uniform(-0.3, 0.3, (n_levels, 1 << log2_table, 2)).astype(np.float32)
    w = (rng.uniform(-1, 1, (5, 64, 64)) * math.sqrt(6 / 64)).astype(np.float32)
    w[4] *= 0.2
    w[4, 3:] = 0
    return table, w


def _prepare_frame(c, seed, rng):
    sc = _scene(rng, c["width"], c["height"], c["tris"], c["lights"], c["hdr"], c["glass"])
    r = R.Renderer(c["width"], c["height"], grid_res=c["grid"],
                   vox_mode=R.VOX_CONSERVATIVE if c["coverage"] == "sat" else R.VOX_REF_RASTER2X,
                   mip_mode={"aniso": R.MIP_ANISO, "iso": R.MIP_ISO, "both": R.MIP_BOTH}[c["mips"]],
                   storage=R.STORAGE_RGBA16F if c["hdr"] else R.STORAGE_RGBA8,
                   radiance_max=S.HDR_RADIANCE_MAX if c["hdr"] else 1.0,
                   sampler=R.SAMPLER_EXACT if c["sampler"] == "software" else R.SAMPLER_HW,
                   cone_set=R.CONES_SIX60 if c["cones"] == 6 else R.CONES_REF9, far_share=c["far_share"],
                   overlap_raster=c["overlap"])
    ids = R.load_scene(r, sc)
    r.set_voxel_view_dir(7, 0.0)
    if c["inject"]:
        r.set_light_injection(True)
    st = {"kind": "frame", "r": r, "scene": sc, "ids": ids}
    if c["learned"]:
        # a trained network's parameters (one small step marks it trained; the parameters then come from the seed)
        d = R.mlp_desc(log2_table=17, steps=1, batch=16)
        r.mlp_init(d)
        r.mlp_train_samples(rng.uniform(0.1, 0.9, (16, 12)).astype(np.float32), d)
        r.mlp_set_params(*_network(rng, 17))
        r.set_mlp_judge(16, 0.0)
        r.set_diffuse_mode(R.DIFFUSE_MLP)
    if c["read"] == "host":
        st["out"] = np.empty((c["height"], c["width"], 4), np.uint8)
    _render(st)  # a running program has frames behind it: its work lists have their size
    r.synchronize()
    if c["read"] != "host":
        st["frame"] = torch.as_tensor(_DeviceFrame(r), device="cuda")
    return st


def _batch_layout(c):
    """(triangles, width, height, grid, cone set) of each scene of a batch: its layout, not its content."""
    rng = np.random.default_rng(c["layout"])
    grids = [g for g in S.BATCH_GRIDS if g <= c["max_grid"]]
    return [(int(math.exp(rng.uniform(math.log(c["min_tris"]), math.log(c["max_tris"])))),
             *S.BATCH_FRAMES[int(rng.integers(len(S.BATCH_FRAMES)))], grids[int(rng.integers(len(grids)))],
             int(rng.integers(2))) for _ in range(c["scenes"])]


def _prepare_batch(c, seed, rng):
    items = [(_scene(rng, w, h, tris), w, h, grid, cones) for tris, w, h, grid, cones in _batch_layout(c)]
    b = R.Batch(items, use_graph=True)
    b.render()
    b.synchronize()
    return {"kind": "batch", "b": b, "items": items}


def _prepare_voxelize(c, seed, rng):
    sc = _scene(rng, 256, 256, c["tris"], c["lights"])
    keep, meshes = [], []
    for mesh, model in zip(sc.meshes, sc.models):
        t = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
             for x in (mesh.verts, mesh.indices.view(np.int32), mesh.tri_material().view(np.int32))]
        keep.append(t)
        m = R.DeviceMesh(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), mesh.verts.shape[0], mesh.n_tris)
        m.model[:] = [float(x) for x in model]
        meshes.append(m)
    mats = torch.from_numpy(sc.materials.view(np.uint8).reshape(-1).copy()).cuda()
    out = torch.empty((c["grid"],) * 3 + (4,), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return {"kind": "voxelize", "meshes": meshes, "keep": keep, "mats": mats, "n_mats": len(sc.materials), "scene": sc,
            "grid": c["grid"], "mode": R.VOX_CONSERVATIVE if c["coverage"] == "sat" else R.VOX_REF_RASTER2X, "out": out}


def _train_rows(rng, n):
    pos = rng.random((n, 3), np.float32) * np.float32(0.96) + np.float32(0.02)
    nrm = rng.standard_normal((n, 3), np.float32)
    alb = rng.random((n, 3), np.float32)
    target = 0.5 + 0.3 * np.sin(6 * pos[:, :1] + 2 * pos[:, 1:2]) * np.cos(4 * pos[:, 2:]) + 0.1 * alb
    return np.concatenate([pos, nrm, alb, target.astype(np.float32)], 1)


def _prepare_train(c, seed, rng):
    r = R.Renderer(16, 16, grid_res=16)
    desc = R.mlp_desc(log2_table=c["log2_table"], steps=c["steps"], batch=c["batch"], lr=1e-4)
    return {"kind": "train", "r": r, "desc": desc, "rows": _train_rows(rng, c["rows"]),
            "params": _network(rng, c["log2_table"]), "log2": c["log2_table"]}


# --------------------------------------------------------------------- run ----
def _render(st):
    r, sc = st["r"], st["scene"]
    r.set_camera_transform(sc.view, sc.proj)
    R.queue_scene(r, sc, st["ids"])
    r.render()


def run(st):
    if st["kind"] == "frame":
        _render(st)
        if "out" in st:
            return st["r"].read_frame(R.FRAME_RGBA8, out=st["out"])
        return st["frame"]
    if st["kind"] == "batch":
        st["b"].render()
        return [st["b"].read_frame(i) for i in range(len(st["items"]))]
    if st["kind"] == "voxelize":
        R.voxelize_noalloc(st["meshes"], st["mats"].data_ptr(), st["n_mats"], st["scene"].lights, st["scene"].cube_size,
                           st["grid"], st["mode"], st["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return st["out"]
    # a training job: the optimiser's state cleared, the checkpoint's parameters, the steps, what came of them
    r = st["r"]
    r.mlp_init(st["desc"])
    r.mlp_set_params(*st["params"])
    rep = r.mlp_train_samples(st["rows"], st["desc"])
    table, w = r.mlp_get_params(log2_table=st["log2"])
    return {"table": table, "weights": w, "loss": np.array([rep["loss_first"], rep["loss_last"]], np.float32)}


# -------------------------------------------------------------------- work ----
# Two-level texture lookups of a pixel (each 16 texels of 4 channels: 128 multiply-adds' worth of flops),
# as counted on the headline frame: the learned frame has no diffuse cones, the per-pixel one all of them.
_LOOKUP_FLOPS = 128.0


def _steps(grid, aperture, reach):
    """March steps of a cone: three voxels out, then half the diameter (one voxel at least) at a time."""
    v, d, n = 1.0 / grid, 3.0 / grid, 0
    while d < reach:
        d += max(0.5 * d * aperture, v)
        n += 1
    return n


def _maps_bytes(grid, mips, texel):
    chain = sum((grid >> l) ** 3 for l in range(1, min(7, grid.bit_length())))
    return texel * (grid ** 3 + chain * {"aniso": 6, "iso": 1, "both": 7}[mips])


def _frame_work(w, h, grid, tris, cones, mips, texel, shared, diffuse, lights, inject=False):
    px = w * h
    fetch = 1 if mips == "iso" else 3
    aperture = 1.1547 if cones == 6 else 0.5579
    per_px = lights * 0.2 * _steps(grid, 0.1, 0.5) * fetch + _steps(grid, 1.0, 0.6) * fetch
    if diffuse:
        n = _steps(grid, aperture, 0.6)
        per_px += cones * fetch * ((1 + (n - 1) / 8.0) if shared else n)
    maps = _maps_bytes(grid, mips, texel)
    geometry = tris * (12 + 4 + 16)  # indices, draw object, half a vertex a triangle
    return {"bytes": float(geometry + 2 * maps + 4 * px + (12 * grid ** 3 if inject else 0)),
            "flops": float(px * per_px * _LOOKUP_FLOPS)}


def work(case):
    c = case
    if c["kind"] == "frame":
        w = _frame_work(c["width"], c["height"], c["grid"], c["tris"], c["cones"], c["mips"], 8 if c["hdr"] else 4,
                        c["far_share"] and c["sampler"] == "texture", not c["learned"], c["lights"], c["inject"])
        if c["learned"]:
            w["flops"] += c["width"] * c["height"] * 2.0 * (4 * 64 * 64 + 3 * 64)
        return w
    if c["kind"] == "batch":
        each = [_frame_work(w, h, grid, tris, 6 if cones else 9, "aniso", 4, True, True, 1)
                for tris, w, h, grid, cones in _batch_layout(c)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if c["kind"] == "voxelize":
        return {"bytes": float(c["tris"] * 32 + 4 * c["grid"] ** 3), "flops": float(c["tris"] * 400)}
    n = min(c["batch"], c["rows"])
    params = 16 * (2 << c["log2_table"]) + 5 * 4096
    per_row = 3 * 2.0 * (4 * 64 * 64 + 3 * 64) + 16 * 8 * 8
    return {"bytes": float(c["rows"] * 48 + c["steps"] * (n * 48 + params * 32)), "flops": float(c["steps"] * n * per_row)}


def exact(case, seed):
    """None: frames and voxels are bytes, and the parameters after several steps of an optimiser that divides by
    the gradients' own size have no value that arithmetic in another width would meet."""
    return None
