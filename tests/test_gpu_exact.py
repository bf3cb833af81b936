"""The plain forms' traversals on the optimised structures (compute-only
frames, G-buffer, deferred resolve, any hit) against the reference walks they
stand for: bit for bit, tolerance zero.  The same call takes either path: a
context without prepared structures answers its first rays (200,000, and 400
more an object) with the reference walk, a prepared one none.  Scenes with
coincident surfaces, shared edges under rays aimed at vertices and edges,
axis-parallel rays, grazing rays, thin triangles, scaled and mirrored
looks from far outside, analytic shapes, textures and refits."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu


def crowd(entities, lib, cfg, name):
    """A scene with far-away extra objects, so that small images stay on the
    reference walk until the structures are prepared."""
    h = lib.add(*scenes.box_mesh((0.1, 0.1, 0.1)))
    far = [scenes.entity(_lib.SHAPE_MESH, _lib.MAT_LAMBERTIAN, (500.0 + k % 20, 500.0 + k // 20, 500.0), mesh=h)
           for k in range(400)]
    return scenes._finish(list(entities) + far, lib, cfg, name)


def field(ggx=False):
    return scenes.wavefront_scene(seed=9, width=96, height=64, depth=5, n_meshes=6, n_instances=300, n_lights=5,
                                  target_tris=30_000, ggx=ggx)


def boxes():
    """Cubes stacked face to face on a floor, thin slivers, analytic shapes."""
    lib = scenes.MeshLibrary()
    cube, floor = lib.add(*scenes.box_mesh((1, 1, 1))), lib.add(*scenes.quad_mesh((0, 0, 40), (40, 0, 0)))
    v, i = scenes.icosphere(3, 1.5)
    v = v.copy()
    v["py"] *= 0.002  # slivers
    flat = lib.add(v, i)
    L = _lib
    ents = [scenes.entity(L.SHAPE_QUAD, L.MAT_DIFFUSE_LIGHT, (-3, 12, -3), emission=15.0, u=(6.0, 0, 0), v=(0, 0, 6.0)),
            scenes.entity(L.SHAPE_SPHERE, L.MAT_DIELECTRIC, (3.0, 1.0, 3.0), radius=1.0, ior=1.5),
            scenes.entity(L.SHAPE_SPHERE, L.MAT_METAL, (-3.0, 1.0, 4.0), radius=1.0, fuzz=0.1, albedo=(0.8, 0.7, 0.6)),
            scenes.entity(L.SHAPE_BOX, L.MAT_LAMBERTIAN, (5.0, 1.0, -3.0), half_extent=(1, 1, 1), albedo=(0.4, 0.5, 0.6)),
            scenes.entity(L.SHAPE_BOX, L.MAT_LAMBERTIAN, (-5.0, 1.0, -3.0), half_extent=(1, 1, 1), rotation=scenes.yaw_quat(0.4),
                          albedo=(0.6, 0.5, 0.4)),
            scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (0, 0, 0), mesh=floor, albedo=(0.5, 0.5, 0.5))]
    for x in range(-2, 3):
        for y in range(3):
            ents.append(scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (2.0 * x, 1.0 + 2.0 * y, -6.0), mesh=cube,
                                      albedo=(0.3 + 0.1 * x, 0.5, 0.4)))
    ents.append(scenes.entity(L.SHAPE_MESH, L.MAT_METAL, (0, 3, 2), mesh=flat, fuzz=0.0, rotation=scenes.yaw_quat(0.3),
                              scale=0.7, albedo=(0.9, 0.9, 0.9)))
    cfg = scenes.make_config(96, 64, (0, 5, 20), (0, 2, 0), depth=5, sky=(0.3, 0.4, 0.5))
    return crowd(ents, lib, cfg, "boxes")


def test_rays(s, n, seed):
    """Random segments, half of them aimed at vertices, edge midpoints or along
    axes."""
    rng = np.random.default_rng(seed)
    ins = s.instances[rng.integers(0, len(s.instances), n)]
    tri = (rng.random(n) * ins["triangleCount"]).astype(np.int64)
    corner = s.indices[ins["indexBase"] + 3 * tri + rng.integers(0, 3, n)] + ins["vertexBase"]
    other = s.indices[ins["indexBase"] + 3 * tri] + ins["vertexBase"]
    v = s.vertices
    p = np.stack([v[a][corner] for a in ("px", "py", "pz")], 1).astype(np.float64)
    q = np.stack([v[a][other] for a in ("px", "py", "pz")], 1).astype(np.float64)
    local = np.where(rng.random((n, 1)) < 0.5, p, 0.5 * (p + q))
    k = np.where(ins["scale"] == 0, 1.0, ins["scale"])[:, None]
    u = np.stack([ins[a] for a in ("qx", "qy", "qz")], 1).astype(np.float64)
    t = 2 * np.cross(u, local * k)
    world = local * k + ins["qw"][:, None] * t + np.cross(u, t) + np.stack([ins[a] for a in ("px", "py", "pz")], 1)
    o = world + rng.normal(size=(n, 3)) * rng.choice([0.01, 1.0, 30.0, 300.0], (n, 1))
    d = world - o
    loose = rng.random(n) < 0.4
    d[loose] += rng.normal(size=(loose.sum(), 3)) * 0.1 * np.linalg.norm(d[loose], axis=1, keepdims=True)
    axis = rng.random(n) < 0.1
    d[axis] = np.eye(3)[rng.integers(0, 3, axis.sum())] * rng.choice([-1.0, 1.0], (axis.sum(), 1))
    dist = np.linalg.norm(d, axis=1)
    d /= dist[:, None]
    r = np.zeros(n, _lib.RAY)
    for j, x in enumerate("xyz"):
        r["o" + x], r["d" + x] = o[:, j], d[:, j]
    r["tnear"], r["time"] = 0.001, 0.25
    return r, (dist * rng.choice([0.5, 1.0, 1.0 + 1e-6, 2.0], n)).astype(np.float32)


test_rays.__test__ = False


def both_any_hits(s, rays, tmax):
    """(exact walk, reference walk): a prepared context, and contexts that are
    asked too little to prepare."""
    with Context(96, 64) as ctx:
        ctx.upload(s)
        ctx.prepare_fast()
        got = ctx.any_hit(rays, tmax)
    want = []
    for k in range(0, len(rays), 150_000):
        with Context(96, 64) as ctx:
            ctx.upload(s)
            want.append(ctx.any_hit(rays[k:k + 150_000], tmax[k:k + 150_000]))
    return got, np.concatenate(want)


@pytest.mark.parametrize("scene", [field, boxes])
def test_any_hit(scene):
    s = scene()
    n = 400_000
    rays, tmax = test_rays(s, n, 5)
    got, want = both_any_hits(s, rays, tmax)
    assert np.array_equal(got, want)
    assert 0.05 < want.mean() < 0.99


def test_any_hit_of_odd_rays():
    """NaN, infinite, zero, negative and huge values in rays and bounds."""
    s = boxes()
    n = 300 * len(s.objects)
    rays, tmax = test_rays(s, n, 6)
    rng = np.random.default_rng(7)
    odd = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, -5.0, 1e-42, 1e30, -1e30, 3e38], np.float32)
    for f in ("ox", "oy", "oz", "tnear", "dx", "dy", "dz", "time"):
        pick = rng.random(n) < 0.08
        rays[f][pick] = rng.choice(odd, pick.sum())
    pick = rng.random(n) < 0.1
    tmax[pick] = rng.choice(odd, pick.sum())
    got, want = both_any_hits(s, rays, tmax)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("scene,frames", [(field, 3), (lambda: field(True), 3), (boxes, 6)])
def test_compute_only_frames(scene, frames):
    s = scene()
    out = []
    for prepared in (False, True):
        with Context(96, 64) as ctx:
            ctx.upload(s)
            if prepared:
                ctx.prepare_fast()
            cfg = s.config.copy()
            for k in range(frames):
                cfg["batch"] = k
                ctx.set_config(cfg)
                ctx.render_frame(_lib.MODE_COMPUTE_ONLY)
            out.append((ctx.read_image(_lib.IMAGE_ACCUM), ctx.read_image(_lib.IMAGE_DISPLAY)))
    assert np.array_equal(out[0][0].view(np.uint8), out[1][0].view(np.uint8))
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("scene", [field, boxes])
@pytest.mark.parametrize("scale", [1.0, 0.75])
def test_hybrid_frames_and_refit(scene, scale):
    s = scene()
    rng = np.random.default_rng(3)
    poses = [None, scenes.random_walk(s.instances, rng), scenes.random_walk(s.instances, rng, step=3.0, angle=1.0)]
    out = []
    for prepared in (False, True):
        images = []
        with Context(96, 64, hybrid=True) as ctx:
            ctx.upload(s)
            cfg = s.config.copy()
            cfg["traceScale"], cfg["depth"] = scale, 3
            for k, pose in enumerate(poses):
                if pose is not None:
                    ctx.refit_instances(pose)
                if prepared:
                    ctx.prepare_fast()
                cfg["frameIndex"], cfg["historyReset"] = k, 1 if k == 0 else 0
                ctx.set_config(cfg)
                ctx.build_gbuffer()
                ctx.render_frame(_lib.MODE_DEFERRED)
                images += list(ctx.read_planes()) + [ctx.read_deferred_accum(), ctx.read_image(_lib.IMAGE_DISPLAY)]
        out.append(images)
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


def test_textures_and_media():
    """Textured shapes on the exact walk; media and moving spheres stay on the
    reference walk and render as before."""
    s = scenes.textured_box(width=96, height=64)
    m = scenes.media_box(width=96, height=64)
    for scene in (s, m):
        out = []
        for samples in (1, 4):  # one call of 4 samples equals its own repetition
            with Context(96, 64) as ctx:
                ctx.upload(scene)
                cfg = scene.config.copy()
                cfg["samples"] = 4
                for _ in range(samples):
                    ctx.set_config(cfg)
                    ctx.render_frame(_lib.MODE_COMPUTE_ONLY)
                out.append(ctx.read_image(_lib.IMAGE_ACCUM))
        assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("scene", [field, boxes, lambda: scenes.cornell_box(width=96, height=64)])
def test_rays_without_a_direction(scene):
    """A direction that is NaN on every axis (a path past a degenerate normal)
    gets the reference walk's answer from every optimised variant."""
    s = scene()
    n = 300
    rays, _ = test_rays(s, n, 8)
    for x in "xyz":
        rays["d" + x] = np.nan
    rays["ox"][::3] = np.nan
    with Context(96, 64) as ctx:
        ctx.upload(s)
        for plain, fast in ((_lib.VARIANT_PLAIN, (_lib.VARIANT_FAST, _lib.VARIANT_FAST_WALK)),
                            (_lib.VARIANT_PLAIN_WT, (_lib.VARIANT_QUANT,))):
            want = ctx.closest_hit(rays, plain)
            for v in fast:
                assert np.array_equal(ctx.closest_hit(rays, v).view(np.uint8), want.view(np.uint8)), v
