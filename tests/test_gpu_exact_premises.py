"""What the exact walks (exact_trace.cuh) count on, at the edges of it: rays
whose reference answer comes from rounding far larger than the scene's boxes
allow for, and uploaded trees and transforms that the reference walk takes as
they are.  Any hit of a prepared context against the reference walk's, bit
for bit (tolerance zero): a scene outside the premises has to keep the
reference walk's answers."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu
L = _lib


def rays_to(origin, points, rng, spread=0.0):
    """Rays from around `origin` through the points; (rays, distance)."""
    n = len(points)
    o = np.asarray(origin, np.float64) + spread * rng.normal(size=(n, 3))
    d = points - o
    dist = np.linalg.norm(d, axis=1)
    d /= dist[:, None]
    r = np.zeros(n, L.RAY)
    for k, x in enumerate("xyz"):
        r["o" + x], r["d" + x] = o[:, k], d[:, k]
    r["tnear"], r["time"] = 0.001, 0.5
    return r, dist


def finish(ents, lib, name):
    return scenes._finish(ents, lib, scenes.make_config(96, 64, (0, 0, 20), (0, 0, 0)), name)


def small_mesh(lib, half=0.001, at=(0.0, 0.0, 0.0)):
    return scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, at, mesh=lib.add(*scenes.box_mesh((half,) * 3)))


def both_any_hits(s, rays, tmax):
    """(on the structures, by the reference walk)"""
    out = []
    for mode in (L.PLAIN_WALK_PREPARED, L.PLAIN_WALK_REFERENCE):
        with scenes_context(s) as ctx:
            ctx.prepare_fast()
            ctx.set_plain_walk(mode)
            out.append(ctx.any_hit(rays, tmax))
    return out


def agree(s, rays, tmax):
    got, want = both_any_hits(s, rays, tmax)
    assert 0 < want.mean() < 1
    assert np.array_equal(got, want)


def limb(rng, centre, radius, n, reach):
    """Points around a sphere's outline as seen along x, out to reach radii."""
    a, k = rng.uniform(0, 2 * np.pi, n), radius * rng.uniform(0.9, reach, n)
    return np.asarray(centre) + np.stack([0 * a, k * np.cos(a), k * np.sin(a)], 1)


def test_tiny_spheres_seen_from_far():
    """Spheres of radius 0.01 from 16 units away: the discriminant's rounding
    is as large as the squared radius."""
    rng = np.random.default_rng(1)
    lib = scenes.MeshLibrary()
    ents = [scenes.entity(L.SHAPE_SPHERE, L.MAT_LAMBERTIAN, (0, y, z), radius=0.01)
            for y, z in ((-0.04, -0.04), (0.04, 0.04))] + [small_mesh(lib)]
    s = finish(ents, lib, "tiny spheres")
    p = np.concatenate([limb(rng, (0, y, z), 0.01, 60_000, 1.6) for y, z in ((-0.04, -0.04), (0.04, 0.04))])
    rays, dist = rays_to((15.9, 0.01, 0.02), p, rng, 0.005)
    agree(s, rays, (dist + 1.0).astype(np.float32))


def test_ground_sphere_with_small_spheres():
    """A ground sphere of radius 1000 under spheres of radius 0.2."""
    rng = np.random.default_rng(2)
    lib = scenes.MeshLibrary()
    at = [(x, 0.2, z) for x in (-3.0, 0.0, 3.0) for z in (-3.0, 0.0, 3.0)]
    ents = [scenes.entity(L.SHAPE_SPHERE, L.MAT_LAMBERTIAN, (0, -1000, 0), radius=1000.0)]
    ents += [scenes.entity(L.SHAPE_SPHERE, L.MAT_LAMBERTIAN, a, radius=0.2) for a in at] + [small_mesh(lib, 0.1, (0, 2, 0))]
    s = finish(ents, lib, "ground sphere")
    p = np.concatenate([limb(rng, a, 0.2, 12_000, 1.5) for a in at])
    origin = np.array([(12.0, 0.5, 1.0), (900.0, 3.0, 20.0), (90.0, 0.4, 5.0)])[rng.integers(0, 3, len(p))]
    rays, dist = rays_to(origin, p, rng, 0.05)
    agree(s, rays, (dist * rng.choice([0.9, 2.0], len(p))).astype(np.float32))


def test_refit_that_grows_the_scene():
    """Spheres of radius 0.5 in a scene of 5 units whose mesh a refit moves
    1,000 away, and rays from there."""
    rng = np.random.default_rng(3)
    lib = scenes.MeshLibrary()
    at = [(0, -2.0, -2.0), (0, 2.0, 2.0)]
    ents = [scenes.entity(L.SHAPE_SPHERE, L.MAT_LAMBERTIAN, a, radius=0.5) for a in at] + [small_mesh(lib, 0.5)]
    s = finish(ents, lib, "refit")
    pose = s.instances.copy()
    pose["px"] = 1000.0
    p = np.concatenate([limb(rng, a, 0.5, 60_000, 2.0) for a in at])
    rays, dist = rays_to((6000.0, 0.3, 0.2), p, rng, 0.2)
    tmax = (dist * 2.0).astype(np.float32)
    got = []
    for prepared in (True, False):
        with scenes_context(s) as ctx:
            if prepared:
                ctx.prepare_fast()
            ctx.refit_instances(pose)
            if prepared:
                ctx.prepare_fast()
            got.append(ctx.any_hit(rays, tmax))
    assert 0 < got[1].mean() < 1
    assert np.array_equal(*got)


def scenes_context(s):
    ctx = Context(96, 64)
    ctx.upload(s)
    ctx.set_plain_walk(L.PLAIN_WALK_PREPARED)
    return ctx


def test_boxes_beside_a_ground_sphere():
    """The widening is the exact walks' own: the boxes that every optimised walk
    shares stay the objects' (an instance-tree leaf or two a camera ray on a
    plain of small spheres, all 400 of them when the boxes were widened by the
    scene's reach)."""
    import ctypes
    import torch
    rng = np.random.default_rng(8)
    lib = scenes.MeshLibrary()
    ents = [scenes.entity(L.SHAPE_SPHERE, L.MAT_LAMBERTIAN, (0, -1000, 0), radius=1000.0)]
    ents += [scenes.entity(L.SHAPE_SPHERE, L.MAT_LAMBERTIAN, (x + 0.9 * rng.random(), 0.2, z + 0.9 * rng.random()), radius=0.2)
             for x in range(-10, 10) for z in range(-10, 10)] + [small_mesh(lib, 0.5, (0, 1, 0))]
    s = scenes._finish(ents, lib, scenes.make_config(96, 64, (13, 2, 3), (0, 0, 0)), "plain of spheres")
    with scenes_context(s) as ctx:
        ctx.prepare_fast()
        n = 96 * 64
        rays = torch.from_numpy(ctx.camera_rays().view(np.uint8)).cuda()
        count = np.zeros(6, np.uint64)
        L.check(L.lib().ae_trace_counters_variant(ctx.handle, ctypes.c_void_p(rays.data_ptr()), n, L.VARIANT_FAST,
                                                  L.ptr(count)), ctx.handle)
        assert count[1] < 10 * n


@pytest.mark.parametrize("shape", [L.SHAPE_QUAD, L.SHAPE_TRIANGLE])
@pytest.mark.parametrize("width", [1e-4, 5e-3])
def test_skewed_planar_objects(shape, width):
    """Edges nearly parallel (shape factors of 100,000 and 2,000): the normal's
    rounding tilts the plane, and rays are accepted far off the shape."""
    rng = np.random.default_rng(4)
    lib = scenes.MeshLibrary()
    a = rng.normal(size=3)
    a /= np.linalg.norm(a)
    b = np.cross(a, rng.normal(size=3))
    b /= np.linalg.norm(b)
    u, v = 10.0 * a, 9.0 * a + width * b
    at = np.array([(-4.0, -3.0, -5.0), (3.0, 4.0, 5.0)])
    ents = [scenes.entity(shape, L.MAT_LAMBERTIAN, p, u=tuple(u), v=tuple(v)) for p in at] + [small_mesh(lib)]
    s = finish(ents, lib, "skewed")
    n = 140_000
    away = 1.5 * rng.uniform(-1, 1, (n, 2)) ** 5
    p = at[rng.integers(0, 2, n)] + rng.uniform(0, 19, (n, 1)) * a + away[:, :1] * np.cross(a, b) + away[:, 1:] * b
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays, dist = rays_to(p - rng.choice([3.0, 30.0, 300.0], (n, 1)) * d, p, rng)
    agree(s, rays, (dist * 1.5).astype(np.float32))


@pytest.mark.parametrize("norm", [0.9995, 1.0005, 0.9, 1.0 + 1e-7])
def test_quaternions_off_unit_length(norm):
    """The walks' transform to a mesh's space uses the conjugate, which is the
    inverse of a unit quaternion only."""
    rng = np.random.default_rng(5)
    lib = scenes.MeshLibrary()
    ents = [scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (0, 0, 0), rotation=scenes.yaw_quat(np.pi / 2),
                          mesh=lib.add(*scenes.box_mesh((5, 5, 5)))),
            scenes.entity(L.SHAPE_QUAD, L.MAT_LAMBERTIAN, (-8, -8, -8), u=(1.0, 0, 0), v=(0, 1.0, 0)),
            scenes.entity(L.SHAPE_QUAD, L.MAT_LAMBERTIAN, (7, 7, 8), u=(1.0, 0, 0), v=(0, 1.0, 0))]
    s = finish(ents, lib, "quaternion")
    for q in ("qx", "qy", "qz", "qw"):
        s.instances[q] *= np.float32(norm)
    n = 140_000
    # Points in the outermost shell of the box, seen almost along its faces.
    grow = 1.0 / norm ** 2 if norm < 1 else 1.0
    p = rng.uniform(-5, 5, (n, 3))
    axis = rng.choice([0, 2], n)
    p[np.arange(n), axis] = rng.choice([-1.0, 1.0], n) * 5.0 * rng.uniform(min(grow, 1.0) - 2e-4, max(grow, 1.0) + 1.5e-3, n)
    side = np.stack([np.where(axis == 0, 0.0, 1.0), rng.normal(size=n) * 0.2, np.where(axis == 0, 1.0, 0.0)], 1)
    rays, dist = rays_to(p - 25.0 * side, p, rng, 1e-3)
    agree(s, rays, (dist * 2.0).astype(np.float32))


@pytest.mark.parametrize("what", ["far", "nan place", "nan scale", "tiny scale", "quad", "nan quad", "box", "angle"])
def test_transforms_that_are_no_plain_numbers(what):
    """One instance or object at infinity, NaN, inside out or turned by many
    radians: the reference walk goes on with the others, and hits the odd one
    where its arithmetic says so."""
    rng = np.random.default_rng(11)
    lib = scenes.MeshLibrary()
    ents = [scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (0, 0, 0), mesh=lib.add(*scenes.box_mesh((3, 3, 3)))),
            scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (7, 0, 0), mesh=lib.add(*scenes.box_mesh((1, 2, 1)))),
            scenes.entity(L.SHAPE_QUAD, L.MAT_LAMBERTIAN, (-8, -8, -8), u=(6.0, 0, 0), v=(0, 6.0, 0)),
            scenes.entity(L.SHAPE_BOX, L.MAT_LAMBERTIAN, (0, 8, 0), half_extent=(1, 2, 3))]
    s = finish(ents, lib, "odd")
    odd = np.argmax(s.instances["px"])
    quad, box = (np.flatnonzero(s.objects["shapeType"] == k)[0] for k in (L.SHAPE_QUAD, L.SHAPE_BOX))
    if what == "far":
        s.instances["px"][odd] = np.inf
    elif what == "nan place":
        s.instances["py"][odd] = np.nan
    elif what == "nan scale":
        s.instances["scale"][odd] = np.nan
    elif what == "tiny scale":
        s.instances["scale"][odd] = 1e-30
    elif what == "quad":
        s.objects["x"][quad] = np.inf
    elif what == "nan quad":
        s.objects["y"][quad] = np.nan
    elif what == "box":
        s.objects["half_y"][box] *= -1
    else:
        s.objects["rotation"][box] = 1e7
    p = rng.uniform(-9, 9, (60_000, 3))
    rays, dist = rays_to(p + 15.0 * rng.normal(size=p.shape), p, rng)
    agree(s, rays, (dist * 2.0).astype(np.float32))


def test_refit_to_infinity_and_back():
    """An instance hidden by moving it to infinity, and shown again."""
    rng = np.random.default_rng(12)
    lib = scenes.MeshLibrary()
    ents = [scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (x, 0, 0), mesh=lib.add(*scenes.box_mesh((2, 2, 2))))
            for x in (-4, 4)]
    s = finish(ents, lib, "hidden")
    hidden = s.instances.copy()
    hidden["px"][1] = np.inf
    p = rng.uniform(-7, 7, (40_000, 3))
    rays, dist = rays_to(p + 12.0 * rng.normal(size=p.shape), p, rng)
    tmax = (dist * 2.0).astype(np.float32)
    answers = []
    for mode in (L.PLAIN_WALK_PREPARED, L.PLAIN_WALK_REFERENCE):
        with scenes_context(s) as ctx:
            ctx.set_plain_walk(mode)
            for pose in (hidden, s.instances, hidden):
                ctx.refit_instances(pose)
                ctx.prepare_fast()
                answers.append(ctx.any_hit(rays, tmax))
            ctx.refit_instances(s.instances)
            ctx.prepare_fast()
            answers.append(ctx.any_hit(rays, tmax))
            assert ctx.plain_walk_used() == (mode == L.PLAIN_WALK_PREPARED)
    for a, b in zip(answers[:4], answers[4:]):
        assert 0 < b.mean() < 1 and np.array_equal(a, b)


def test_refit_to_quaternions_off_unit_length():
    """The same by a refit, and back."""
    rng = np.random.default_rng(9)
    lib = scenes.MeshLibrary()
    ents = [scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (0, 0, 0), rotation=scenes.yaw_quat(np.pi / 2),
                          mesh=lib.add(*scenes.box_mesh((5, 5, 5)))),
            scenes.entity(L.SHAPE_QUAD, L.MAT_LAMBERTIAN, (-8, -8, -8), u=(16.0, 0, 0), v=(0, 1.0, 0)),
            scenes.entity(L.SHAPE_QUAD, L.MAT_LAMBERTIAN, (7, 7, 8), u=(1.0, 0, 0), v=(0, 1.0, 0))]
    s = finish(ents, lib, "quaternion")
    off = s.instances.copy()
    for q in ("qx", "qy", "qz", "qw"):
        off[q] *= np.float32(0.95)
    n = 60_000
    p = rng.uniform(-6.2, 6.2, (n, 3))
    rays, dist = rays_to(p + 25.0 * rng.normal(size=(n, 3)), p, rng)
    tmax = (dist * 2.0).astype(np.float32)
    got = []
    for prepared in (True, False):
        answers = []
        for pose in (off, s.instances):
            with scenes_context(s) as ctx:
                if prepared:
                    ctx.prepare_fast()
                ctx.refit_instances(off)
                if pose is not off:
                    ctx.refit_instances(pose)
                if prepared:
                    ctx.prepare_fast()
                answers.append(ctx.any_hit(rays, tmax))
        got.append(answers)
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert not np.array_equal(got[1][0], got[1][1])


@pytest.mark.parametrize("what", ["nodes", "leaves", "root leaf"])
def test_trees_that_do_not_enclose(what):
    """BLAS boxes smaller than what lies below them cut hits off in the
    reference walk."""
    rng = np.random.default_rng(6)
    lib = scenes.MeshLibrary()
    mesh = scenes.icosphere(3, 4.0)
    if what == "root leaf":
        mesh = (mesh[0], mesh[1][:6])
    ents = [scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (0, 0, 0), mesh=lib.add(*mesh)),
            scenes.entity(L.SHAPE_QUAD, L.MAT_LAMBERTIAN, (-8, -8, -8), u=(16.0, 0, 0), v=(0, 1.0, 0))]
    s = finish(ents, lib, "loose tree")
    b = s.blas
    assert (len(b) == 1) == (what == "root leaf")
    pick = b["count"] == 0 if what == "nodes" else b["count"] > 0
    if what == "nodes":
        pick[0] = False
    for x in "xyz":
        mid = 0.5 * (b["min_" + x] + b["max_" + x])
        b["min_" + x][pick] = (mid + 0.6 * (b["min_" + x] - mid))[pick]
        b["max_" + x][pick] = (mid + 0.6 * (b["max_" + x] - mid))[pick]
    p = rng.normal(size=(100_000, 3))
    p *= 4.0 * rng.uniform(0.2, 1.0, (len(p), 1)) / np.linalg.norm(p, axis=1, keepdims=True)
    if what == "root leaf":
        tri = np.stack([mesh[0][x][mesh[1]] for x in ("px", "py", "pz")], 1).astype(np.float64).reshape(-1, 3, 3)
        w = rng.dirichlet((1, 1, 1), len(p))
        p = np.einsum("nk,nkc->nc", w, tri[rng.integers(0, len(tri), len(p))])
    rays, dist = rays_to((3.0, 5.0, 14.0), p, rng, 2.0)
    agree(s, rays, (dist * 1.2).astype(np.float32))


def test_two_meshes_on_one_tree():
    """A tree that two meshes name and that holds one of them only."""
    rng = np.random.default_rng(10)
    lib = scenes.MeshLibrary()
    v, i = scenes.icosphere(3, 3.0)
    small = lib.add(v, i)
    w = v.copy()
    for x in ("px", "py", "pz"):
        w[x] *= 1.4
    big = lib.add(w, i)
    ents = [scenes.entity(L.SHAPE_MESH, L.MAT_LAMBERTIAN, (x, 0, 0), mesh=m) for x, m in ((-6, small), (6, big))]
    ents.append(scenes.entity(L.SHAPE_QUAD, L.MAT_LAMBERTIAN, (-12, -8, -8), u=(24.0, 0, 0), v=(0, 1.0, 0)))
    s = finish(ents, lib, "two meshes")
    assert len(s.instances) == 2
    s.instances["blasBase"] = s.instances["blasBase"].min()
    p = rng.normal(size=(100_000, 3))
    p *= 4.2 * rng.uniform(0.2, 1.0, (len(p), 1)) / np.linalg.norm(p, axis=1, keepdims=True)
    p[:, 0] += rng.choice([-6.0, 6.0], len(p))
    rays, dist = rays_to((3.0, 5.0, 20.0), p, rng, 2.0)
    agree(s, rays, (dist * 1.2).astype(np.float32))
