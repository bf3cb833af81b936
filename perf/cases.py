"""The work a user of the library has it do, as measurable cases.

Six kinds, each through the public entry points:

  rays     closest hit of a batch of rays: picking and sensor queries (host
           arrays), camera rays and diffuse bounces that already lie on the
           device, page-locked host batches
  occlude  any hit of a batch of segments (visibility and light queries)
  frame    progressive frames of one camera: the compute-only form, the
           wavefront form and its precision form; the image is read back once
           the frames are accumulated
  hybrid   interactive frames of the hybrid renderer: G-buffer, deferred
           resolve, temporal upsample, the display image of every frame
  moving   an animated scene: every instance moves, the scene is refit, a
           frame is rendered and shown
  build    acceleration structures of new meshes, device arrays in and out

Scenes are the repository's own generators (aviatorengine2_b200/scenes.py):
the Cornell box, the instanced-mesh scene of the closest-hit benchmark and the
lit instance field of the wavefront benchmark, at their full instance counts
and at smaller triangle budgets.
"""
import ctypes
import math

import numpy as np
import torch

from aviatorengine2_b200 import _lib, scenes
from aviatorengine2_b200.renderer import Context, Renderer, RendererSettings

VARIANTS = {"fast": _lib.VARIANT_FAST, "quant": _lib.VARIANT_QUANT, "walk": _lib.VARIANT_FAST_WALK}
MODES = {"compute": _lib.MODE_COMPUTE_ONLY, "wavefront": _lib.MODE_WAVEFRONT,
         "precision": _lib.MODE_WAVEFRONT_PRECISION}
DEVICE = "cuda"


def listed():
    return [
        # An editor's marquee pick or a small lidar sweep: a few rays, one call.
        {"name": "pick", "kind": "rays", "scene": "cornell", "rays": "scatter", "n": 1000, "variant": "fast",
         "where": "host"},
        # The closest-hit benchmark's two sets: every pixel of a 1080p image,
        # and one diffuse bounce of each.
        {"name": "camera_1080p", "kind": "rays", "scene": "instances", "grid": 512, "instances": 64, "width": 1920,
         "height": 1080, "rays": "camera", "variant": "fast", "where": "device"},
        {"name": "bounce_1080p", "kind": "rays", "scene": "instances", "grid": 512, "instances": 64, "width": 1920,
         "height": 1080, "rays": "bounce", "variant": "walk", "where": "device"},
        # A sensor simulation that keeps its rays in page-locked host memory:
        # unordered rays, an odd count.
        {"name": "sensor_host", "kind": "rays", "scene": "instances", "grid": 256, "instances": 200,
         "rays": "scatter", "n": 300_001, "variant": "walk", "where": "pinned"},
        # Visibility queries of a simulation: segments between random points.
        {"name": "visibility", "kind": "occlude", "scene": "instances", "grid": 256, "instances": 200, "n": 200_003},
        # The reference's own setting: the Cornell box at 320x240, depth 8,
        # 16 progressive frames of the compute-only form.
        {"name": "cornell_preview", "kind": "frame", "scene": "cornell", "width": 320, "height": 240, "depth": 8,
         "mode": "compute", "frames": 16},
        # The reference's default mode, camera and history moving on: small
        # frames of a lit field at three quarters of the trace resolution.
        {"name": "hybrid_540p", "kind": "hybrid", "scene": "field", "tris": 250_000, "instances": 256, "lights": 4,
         "width": 960, "height": 540, "depth": 3, "scale": 0.75, "frames": 2},
        # A thumbnail or a low-latency preview in the wavefront form.
        {"name": "wavefront_thumb", "kind": "frame", "scene": "field", "tris": 250_000, "instances": 256, "lights": 4,
         "ggx": False, "width": 256, "height": 256, "depth": 8, "mode": "wavefront", "frames": 4},
        # The wavefront benchmark's frame: 1024 instances, 16 lights, 12
        # bounces, GGX metal, full HD.
        {"name": "wavefront_1080p", "kind": "frame", "scene": "field", "tris": 2_000_000, "instances": 1024,
         "lights": 16, "ggx": True, "width": 1920, "height": 1080, "depth": 12, "mode": "wavefront", "frames": 1},
        # The precision form at its benchmark setting, accumulated.
        {"name": "precision_540p", "kind": "frame", "scene": "instances", "grid": 512, "instances": 64, "width": 960,
         "height": 540, "depth": 2, "mode": "precision", "frames": 8},
        # A simulation's frame loop: 512 moving instances, one frame a step.
        {"name": "moving_360p", "kind": "moving", "scene": "field", "tris": 500_000, "instances": 512, "lights": 4,
         "ggx": False, "width": 641, "height": 361, "depth": 3, "frames": 2},
        # A level load: the structures of sixteen new meshes.
        {"name": "mesh_build", "kind": "build", "meshes": 16, "tris": 2_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_instances(rng):
    return {"scene": "instances", "grid": rng.choice([96, 128, 192, 256, 384, 512]),
            "instances": _log(rng, 16, 400)}


def _draw_field(rng, tris):
    return {"scene": "field", "tris": _log(rng, 50_000, tris), "instances": _log(rng, 64, 1024),
            "lights": rng.choice([1, 2, 4, 7, 16])}


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "occlude", "frame", "frame", "frame", "hybrid", "moving", "build"])
    case = {"kind": kind}
    if kind == "rays":
        rays = rng.choice(["camera", "bounce", "scatter"])
        if rays == "scatter":
            where = rng.choice(["host", "pinned", "device"])
            case.update({"scene": "cornell"} if rng.random() < 0.3 else _draw_instances(rng))
            case.update({"rays": rays, "n": _log(rng, 500, 1_500_000), "where": where,
                         "variant": rng.choice(["fast", "walk", "quant"])})
        else:
            case.update(_draw_instances(rng))
            w = _log(rng, 200, 1920)
            case.update({"rays": rays, "width": w, "height": max(1, int(w * rng.uniform(0.45, 0.75))),
                         "where": rng.choice(["pinned", "device", "device"]),
                         "variant": rng.choice(["fast", "quant"]) if rays == "camera" else "walk"})
    elif kind == "occlude":
        case.update(_draw_instances(rng))
        case["n"] = _log(rng, 500, 1_000_000)
    elif kind == "frame":
        mode = rng.choice(["compute", "wavefront", "wavefront", "precision"])
        if mode == "compute":
            w = _log(rng, 100, 640)
            case.update({"scene": "cornell", "depth": rng.randint(2, 10), "frames": rng.randint(1, 16)})
        elif rng.random() < 0.3:
            w = _log(rng, 160, 1280)
            case.update(_draw_instances(rng))
            case.update({"depth": rng.randint(1, 4), "frames": rng.randint(1, 8)})
        else:
            w = _log(rng, 160, 1280)
            case.update(_draw_field(rng, 2_000_000))
            case.update({"depth": rng.randint(2, 12), "frames": 1 if w > 500 else rng.randint(1, 4),
                         "ggx": rng.random() < 0.5})
        case.update({"width": w, "height": max(1, int(w * rng.uniform(0.5, 0.8))), "mode": mode})
    elif kind == "hybrid":
        w = _log(rng, 200, 960)
        case.update(_draw_field(rng, 500_000))
        case["lights"] = min(case["lights"], 4)
        case["instances"] = min(case["instances"], 300)
        case.update({"width": w, "height": max(1, int(w * rng.uniform(0.5, 0.7))), "depth": rng.randint(2, 3),
                     "scale": rng.choice([0.5, 0.75, 1.0]), "frames": rng.randint(1, 3)})
    elif kind == "moving":
        w = _log(rng, 160, 800)
        case.update(_draw_field(rng, 1_000_000))
        case["lights"] = min(case["lights"], 4)
        case.update({"width": w, "height": max(1, int(w * rng.uniform(0.5, 0.7))), "depth": rng.randint(1, 4),
                     "frames": rng.randint(1, 3), "ggx": rng.random() < 0.5})
    else:
        case.update({"meshes": _log(rng, 1, 32), "tris": _log(rng, 5_000, 2_000_000)})
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _scene(case, seed):
    w, h = case.get("width", 320), case.get("height", 240)
    if case["scene"] == "cornell":
        return scenes.cornell_box(seed=seed + 1, width=w, height=h, depth=case.get("depth", 8))
    if case["scene"] == "instances":
        g = case["grid"]
        top = max(3, round(math.log2(g)) - 2)
        s = scenes.instanced_meshes(seed=seed + 1, width=w, height=h, levels=(top, top - 1, top - 1, top - 2, top - 2),
                                    grid=g, n_instances=case["instances"], gpu_build=True)
        if case["kind"] == "frame":
            s.config["depth"] = case["depth"]
        return s
    meshes = 16 if case["tris"] < 1_000_000 else 32
    return scenes.wavefront_scene(seed=seed + 1, width=w, height=h, depth=case["depth"], n_meshes=meshes,
                                  n_instances=case["instances"], n_lights=case["lights"], target_tris=case["tris"],
                                  gpu_build=True, ggx=case.get("ggx", False))


def _extent(case):
    """The box that the scene's objects lie in."""
    return (np.array([0.5, 0.5, 0.5]), np.array([9.5, 9.5, 9.5])) if case["scene"] == "cornell" else (
        np.array([0.0, 0.0, 0.0]), np.array([100.0, 100.0, 100.0]))


def _scatter(case, seed, n):
    """Rays from points of the scene in directions of the sphere."""
    rng = np.random.default_rng(seed + 77)
    lo, hi = _extent(case)
    r = np.zeros(n, _lib.RAY)
    o = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    for k, a in enumerate("xyz"):
        r["o" + a], r["d" + a] = o[:, k], d[:, k]
    r["tnear"], r["time"] = 0.001, 0.5
    return r


def _pinned(nbytes):
    return torch.empty(nbytes, dtype=torch.uint8).pin_memory()


def _prepare_rays(case, seed):
    s = _scene(case, seed)
    ctx = Context(case.get("width", 320), case.get("height", 240))
    ctx.upload(s)
    ctx.prepare_fast()
    if case["rays"] == "scatter":
        rays = _scatter(case, seed, case["n"])
    else:
        rays = ctx.camera_rays()
        if case["rays"] == "bounce":
            rays, valid = ctx.bounce_rays(rays, ctx.closest_hit(rays, _lib.VARIANT_FAST))
            # The pixels that hit something, in pixel order; half as many rays
            # as pixels whatever the share of the image that is covered.
            rays = np.resize(rays[valid] if valid.any() else rays, len(rays) // 2)
    n = len(rays)
    state = {"ctx": ctx, "n": n, "variant": VARIANTS[case["variant"]], "where": case["where"]}
    if case["where"] == "device":
        state["rays"] = torch.from_numpy(rays.view(np.float32).reshape(n, 8).copy()).to(DEVICE)
        state["hits"] = torch.zeros(n, 5, dtype=torch.float32, device=DEVICE)
    elif case["where"] == "pinned":
        state["rays"], state["hits"] = _pinned(n * 32), _pinned(n * 20)
        state["rays"].copy_(torch.from_numpy(rays.view(np.uint8).reshape(-1)))
    else:
        state["rays"] = rays
    return state


def _run_rays(s):
    if s["where"] == "device":
        s["ctx"].closest_hit_device(s["rays"].data_ptr(), s["n"], s["hits"].data_ptr(), s["variant"])
        return {"t_alpha_beta": s["hits"][:, :3], "object_prim": s["hits"].view(torch.int32)[:, 3:]}
    if s["where"] == "pinned":
        p = ctypes.c_void_p
        _lib.check(_lib.lib().ae_closest_hit(s["ctx"].handle, p(s["rays"].data_ptr()), s["n"],
                                             p(s["hits"].data_ptr()), s["variant"]), s["ctx"].handle)
        hits = s["hits"].view(torch.float32).view(-1, 5)
        return {"t_alpha_beta": hits[:, :3], "object_prim": hits.view(torch.int32)[:, 3:]}
    hits = s["ctx"].closest_hit(s["rays"], s["variant"])
    flat = hits.view(np.float32).reshape(-1, 5)
    return {"t_alpha_beta": flat[:, :3], "object_prim": flat.view(np.int32)[:, 3:]}


def _prepare_occlude(case, seed):
    s = _scene(case, seed)
    ctx = Context(320, 240)
    ctx.upload(s)
    rng = np.random.default_rng(seed + 99)
    n = case["n"]
    lo, hi = _extent(case)
    a, b = rng.uniform(lo, hi, (n, 3)), rng.uniform(lo, hi, (n, 3))
    dist = np.linalg.norm(b - a, axis=1)
    d = ((b - a) / np.maximum(dist, 1e-6)[:, None]).astype(np.float32)
    r = np.zeros(n, _lib.RAY)
    for k, x in enumerate("xyz"):
        r["o" + x], r["d" + x] = a[:, k].astype(np.float32), d[:, k]
    r["tnear"], r["time"] = 0.001, 0.5
    return {"ctx": ctx, "rays": r, "tmax": (dist - 0.001).astype(np.float32)}


def _prepare_frame(case, seed):
    s = _scene(case, seed)
    if case["mode"] == "compute":
        r = Renderer()
        r.Initialize(RendererSettings(width=case["width"], height=case["height"], hybrid=False))
        r.LoadScene(s)
        return {"renderer": r, "frames": case["frames"]}
    ctx = Context(case["width"], case["height"])
    ctx.upload(s)
    ctx.prepare_fast()
    return {"ctx": ctx, "mode": MODES[case["mode"]], "frames": case["frames"], "config": ctx.get_config().copy()}


def _run_frame(s):
    if "renderer" in s:
        r = s["renderer"]
        r.ResetAccumulation()
        for _ in range(s["frames"]):
            r.RenderFrame()
        return {"accum": r.ctx.read_image(_lib.IMAGE_ACCUM), "display": r.ctx.read_image(_lib.IMAGE_DISPLAY)}
    ctx, cfg = s["ctx"], s["config"]
    for k in range(s["frames"]):
        cfg["batch"] = k
        ctx.set_config(cfg)
        ctx.render_frame(s["mode"])
    return {"accum": ctx.read_image(_lib.IMAGE_ACCUM), "display": ctx.read_image(_lib.IMAGE_DISPLAY)}


def _prepare_hybrid(case, seed):
    s = _scene(case, seed)
    r = Renderer()
    r.Initialize(RendererSettings(width=case["width"], height=case["height"], hybrid=True,
                                  hybridMaxDepth=case["depth"], traceScale=case["scale"]))
    r.LoadScene(s)
    r.config["traceScale"] = case["scale"]
    c = r.config
    rng = np.random.default_rng(seed + 55)
    eye = np.array([c["source_x"], c["source_y"], c["source_z"]], np.float64)
    target = tuple(float(c["target_" + a]) for a in "xyz")
    eyes = [tuple(float(x) for x in eye + rng.normal(0.0, 1.0, 3)) for _ in range(case["frames"])]
    return {"renderer": r, "eyes": eyes, "target": target}


def _run_hybrid(s):
    r = s["renderer"]
    r.ResetAccumulation()
    r.frameIndex = 0
    shown = []
    for eye in s["eyes"]:
        r.SyncCamera(eye, s["target"])
        r.CameraMoved()
        r.ctx.set_config(r.config)
        r.ctx.build_gbuffer()
        r.RenderFrame()
        shown.append(r.ctx.read_image(_lib.IMAGE_DISPLAY))
    return {"shown": shown, "accum": r.ctx.read_deferred_accum()}


def _prepare_moving(case, seed):
    s = _scene(case, seed)
    ctx = Context(case["width"], case["height"])
    ctx.upload(s)
    ctx.prepare_fast()
    rng = np.random.default_rng(seed + 33)
    poses, at = [], s.instances
    for _ in range(case["frames"]):
        at = scenes.random_walk(at, rng)
        poses.append(at)
    return {"ctx": ctx, "poses": poses}


def _run_moving(s):
    ctx, shown = s["ctx"], []
    for pose in s["poses"]:
        ctx.refit_instances(pose)
        ctx.render_frame(_lib.MODE_WAVEFRONT)
        shown.append(ctx.read_image(_lib.IMAGE_DISPLAY))
    return {"shown": shown, "accum": ctx.read_image(_lib.IMAGE_ACCUM)}


def _prepare_build(case, seed):
    rng = np.random.default_rng(seed + 11)
    geometry, _ = scenes.wavefront_meshes(rng, case["meshes"], case["tris"])
    k = len(geometry)
    verts = [torch.from_numpy(v.view(np.float32).reshape(-1, 8).copy()).to(DEVICE) for v, _ in geometry]
    index = [torch.from_numpy(i.astype(np.int32)).to(DEVICE) for _, i in geometry]
    # Spread over the mesh's own scale by the seed, so that no two seeds build the same tree.
    for v in verts:
        v[:, :3] *= torch.tensor(rng.uniform(0.5, 2.0, 3), dtype=torch.float32, device=DEVICE)
    # One allocation for all nodes and one for all reordered indices, each
    # mesh's part on a 256-byte boundary.
    at, parts = [0, 0], []
    for i in index:
        parts.append((at[0], at[1]))
        at = [at[0] + -(-2 * (len(i) // 3) // 16) * 16, at[1] + -(-len(i) // 64) * 64]
    nodes = torch.zeros(at[0], 12, dtype=torch.int32, device=DEVICE)
    ordered = torch.zeros(at[1], dtype=torch.int32, device=DEVICE)
    ptrs = lambda ts: (ctypes.c_void_p * k)(*[t.data_ptr() for t in ts])  # noqa: E731
    return {"k": k, "keep": (verts, index), "nodes": nodes, "ordered": ordered,
            "args": (ptrs(verts), np.array([len(v) for v in verts], np.uint32), ptrs(index),
                     np.array([len(i) for i in index], np.uint32), ptrs([nodes[p:] for p, _ in parts]),
                     np.zeros(k, np.uint32), ptrs([ordered[p:] for _, p in parts]))}


def _run_build(s):
    v, nv, i, ni, n, counts, o = s["args"]
    _lib.check(_lib.lib().ae_mesh_blas_device_many(s["k"], v, _lib.ptr(nv), i, _lib.ptr(ni), n, _lib.ptr(counts), o,
                                                   None), what="ae_mesh_blas_device_many")
    return {"counts": counts.astype(np.int64), "nodes": s["nodes"], "indices": s["ordered"]}


def prepare(case, seed):
    return {"rays": _prepare_rays, "occlude": _prepare_occlude, "frame": _prepare_frame, "hybrid": _prepare_hybrid,
            "moving": _prepare_moving, "build": _prepare_build}[case["kind"]](case, seed) | {"kind": case["kind"]}


def run(state):
    kind = state["kind"]
    if kind == "rays":
        return _run_rays(state)
    if kind == "occlude":
        return {"occluded": state["ctx"].any_hit(state["rays"], state["tmax"])}
    return {"frame": _run_frame, "hybrid": _run_hybrid, "moving": _run_moving, "build": _run_build}[kind](state)


# ---------------------------------------------------------------------------
# The least a pass can do
# ---------------------------------------------------------------------------
def _descent_flops(case):
    """One descent from the root of the instance tree to a triangle: two boxes
    (15 operations each) a level, one transform (60), one triangle (70)."""
    if case["scene"] == "cornell":
        tris, inst = 36, 8
    elif case["scene"] == "instances":
        g = case["grid"]
        top = max(3, round(math.log2(g)) - 2)
        tris = 3 * 2 * (g - 1) ** 2 + sum(20 * 4 ** v for v in (top, top - 1, top - 1, top - 2, top - 2))
        inst = case["instances"]
    else:
        tris, inst = case["tris"], case["instances"]
    return 30.0 * math.log2(max(2, tris / 8 * inst / 4)) + 130.0


def work(case):
    kind = case["kind"]
    if kind == "build":
        # Vertices and indices in; about one node for every triangle and the
        # reordered indices out; a box test against each of a tree's levels.
        t = case["tris"]
        return {"bytes": t * (16.0 + 12.0 + 48.0 + 12.0), "flops": t * 12.0 * math.log2(max(2, t / case["meshes"]))}
    f = _descent_flops(case)
    if kind == "rays":
        px = case.get("width", 0) * case.get("height", 0)
        n = {"scatter": case.get("n"), "camera": px, "bounce": px // 2}[case["rays"]]
        return {"bytes": n * 52.0, "flops": n * f}
    if kind == "occlude":
        return {"bytes": case["n"] * 37.0, "flops": case["n"] * f}
    px = case["width"] * case["height"] * case["frames"]
    if kind == "hybrid":
        traced = px * case["scale"] ** 2
        return {"bytes": px * (36.0 + 2 * 32.0 + 4.0), "flops": px * f + traced * 2 * f}
    # A camera ray and, where the scene has lights, one shadow ray a pixel.
    lit = case["scene"] != "instances"
    return {"bytes": px * 20.0, "flops": px * f * (2 if lit else 1)}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _rotate(q, v):
    """v rotated by the quaternion q (x, y, z, w)."""
    u = q[:3]
    t = 2.0 * np.cross(u, v)
    return v + q[3] * t + np.cross(u, t)


def exact(case, seed):
    """Closest hits of scattered rays in the Cornell box by testing every
    triangle and the light in 64 bits.  Every other case has no closed form
    short of tracing it (millions of triangles, or a path tracer's images)."""
    if case["kind"] != "rays" or case["scene"] != "cornell" or case["rays"] != "scatter" or case["n"] > 200_000:
        return None
    s = _scene(case, seed)
    rays = _scatter(case, seed, case["n"])
    o = np.stack([rays["o" + a] for a in "xyz"], 1).astype(np.float64)
    d = np.stack([rays["d" + a] for a in "xyz"], 1).astype(np.float64)
    surfaces = []
    for obj in s.objects:
        if int(obj["shapeType"]) == _lib.SHAPE_MESH:
            m = s.instances[int(obj["instanceIndex"])]
            q = np.array([m["qx"], m["qy"], m["qz"], m["qw"]], np.float64)
            at = np.array([m["px"], m["py"], m["pz"]], np.float64)
            k = float(m["scale"]) or 1.0
            for t in range(int(m["triangleCount"])):
                ix = s.indices[int(m["indexBase"]) + 3 * t:][:3] + int(m["vertexBase"])
                p = [at + _rotate(q, k * np.array([s.vertices[int(i)][c] for c in ("px", "py", "pz")], np.float64))
                     for i in ix]
                surfaces.append((p[0], p[1] - p[0], p[2] - p[0], True))
        else:
            p = np.array([obj["x"], obj["y"], obj["z"]], np.float64)
            u = np.array([obj["u_x"], obj["u_y"], obj["u_z"]], np.float64)
            v = np.array([obj["v_x"], obj["v_y"], obj["v_z"]], np.float64)
            surfaces.append((p, u, v, False))
    best = np.full(len(o), np.inf)
    out = np.zeros((len(o), 3))
    for p, u, v, tri in surfaces:
        n = np.cross(u, v)
        with np.errstate(divide="ignore", invalid="ignore"):
            t = ((p - o) @ n) / (d @ n)
            w = n / (n @ n)
            x = o + d * t[:, None] - p
            a, b = np.cross(x, v) @ w, np.cross(np.broadcast_to(u, x.shape), x) @ w
        hit = np.isfinite(t) & (t >= 0.001) & (t <= best) & (a >= 0) & (b >= 0)
        hit &= (a + b <= 1) if tri else (a <= 1) & (b <= 1)
        best = np.where(hit, t, best)
        out[hit] = np.stack([t, a, b], 1)[hit]
    return {"t_alpha_beta": torch.from_numpy(out), "object_prim": None}
