"""The optimised walks' structures as the device builds them (4-wide nodes,
triangle records, FP16 shading records), at the sizes where the build can go
wrong: one triangle, a root that is a leaf, few nodes, several hundred meshes,
trees that share binary nodes, and instances that share a tree.  Hits must be
the reference walk's bit for bit (the same triangle test on both sides), so
the tolerance is zero."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu


def rays_through(lo, hi, n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, _lib.RAY)
    a, b = rng.uniform(lo, hi, (n, 3)), rng.uniform(lo, hi, (n, 3))
    d = b - a
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    for k, x in enumerate("xyz"):
        r["o" + x], r["d" + x] = a[:, k], d[:, k]
    r["tnear"] = 0.001
    return r


def check(ctx, rays, label):
    plain = ctx.closest_hit(rays, _lib.VARIANT_PLAIN)
    for v in (_lib.VARIANT_FAST, _lib.VARIANT_FAST_WALK):
        got = ctx.closest_hit(rays, v)
        assert np.array_equal(got.view(np.uint8), plain.view(np.uint8)), (label, v)
    wt = ctx.closest_hit(rays, _lib.VARIANT_PLAIN_WT)
    got = ctx.closest_hit(rays, _lib.VARIANT_QUANT)
    assert np.array_equal(got.view(np.uint8), wt.view(np.uint8)), label
    assert (plain["object"] != _lib.MISS).any(), label


def soup(n, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-4, 4, (n, 1, 3)) + rng.uniform(-1, 1, (n, 3, 3))
    v = np.zeros(3 * n, _lib.VERTEX)
    v["px"], v["py"], v["pz"] = (scale * p).reshape(-1, 3).T
    v["nz"] = 1.0
    return v, np.arange(3 * n, dtype=np.uint32)


@pytest.mark.parametrize("sizes", [[1], [2], [5], [9, 1, 33], [1000, 3, 1025, 64], [7] * 300])
def test_random_meshes(sizes):
    rng = np.random.default_rng(len(sizes) + sizes[0])
    lib = scenes.MeshLibrary()
    ents = []
    for k, n in enumerate(sizes):
        h = lib.add(*soup(n, k, float(rng.choice([1e-3, 1.0, 50.0]) if len(sizes) == 4 else 1.0)))
        at = rng.uniform(-6, 6, 3) if k else np.zeros(3)
        ents.append(scenes.entity(_lib.SHAPE_MESH, _lib.MAT_LAMBERTIAN, at, rotation=scenes.random_quat(rng),
                                  scale=float(rng.uniform(0.5, 2.0)), mesh=h))
    s = scenes._finish(ents, lib, scenes.make_config(64, 48, (0, 0, 20), (0, 0, 0)), "meshes")
    with Context(64, 48) as ctx:
        ctx.upload(s)
        check(ctx, rays_through(-8, 8, 40_000, 3), sizes)


def test_trees_that_share_nodes():
    """Two trees of which the second starts at a node of the first that is a
    4-wide node of both (links are relative to a tree's first node)."""
    v, i = soup(7, 5)
    p = np.stack([v["px"], v["py"], v["pz"]], 1).reshape(7, 3, 3)
    blas = np.zeros(13, _lib.NODE)

    def leaf(at, tri):
        blas[at]["left"], blas[at]["count"] = tri, 1

    def inner(at, left, right, tris):
        blas[at]["left"], blas[at]["right"] = left, right
        box(at, tris)

    def box(at, tris):
        q = p[list(tris)].reshape(-1, 3)
        for k, x in enumerate("xyz"):
            blas[at]["min_" + x], blas[at]["max_" + x] = q[:, k].min() - 0.01, q[:, k].max() + 0.01

    for at, tri in ((2, 0), (3, 1), (4, 2), (9, 3), (10, 4), (11, 5), (12, 6)):
        leaf(at, tri)
        box(at, [tri])
    p[:3] *= 0.1  # the first subtree is the smallest, so that it is not opened
    v["px"], v["py"], v["pz"] = p.reshape(-1, 3).T
    for at, tri in ((2, 0), (3, 1), (4, 2)):
        box(at, [tri])
    inner(0, 1, 6, range(7))
    inner(1, 2, 3, range(3))      # tree 0: leaves 2, 3; tree 1 (from node 1): leaves 3, 4
    inner(6, 7, 8, range(3, 7))
    inner(7, 9, 10, (3, 4))
    inner(8, 11, 12, (5, 6))
    lib = scenes.MeshLibrary()
    h = lib.add(v, i)
    ents = [scenes.entity(_lib.SHAPE_MESH, _lib.MAT_LAMBERTIAN, (x, 0, 0), mesh=h) for x in (-3.0, 3.0)]
    s = scenes._finish(ents, lib, scenes.make_config(64, 48, (0, 0, 20), (0, 0, 0)), "shared")
    s.vertices, s.indices, s.blas = v, i, blas
    s.instances["blasBase"] = [0, 1]
    with Context(64, 48) as ctx:
        ctx.upload(s)
        check(ctx, rays_through(-7, 7, 40_000, 4), "shared nodes")


def test_more_meshes_on_the_same_geometry():
    """A later scene upload that names further meshes of the uploaded
    geometry, and the precision form's shading records with it."""
    lib = scenes.MeshLibrary()
    hs = [lib.add(*scenes.icosphere(3, 1.5)), lib.add(*scenes.box_mesh((1, 2, 1))), lib.add(*soup(50, 8))]
    cfg = scenes.make_config(64, 48, (0, 0, 14), (0, 0, 0), depth=2, sky=(0.5, 0.6, 0.7))

    def scene(n):
        ents = [scenes.entity(_lib.SHAPE_MESH, _lib.MAT_LAMBERTIAN, (3.0 * k - 3.0, 0, 0), mesh=h, albedo=(0.5, 0.6, 0.7))
                for k, h in enumerate(hs[:n])]
        return scenes._finish(ents, lib, cfg, "more")

    one, three = scene(1), scene(3)
    images = []
    for first in (one, three):
        with Context(64, 48) as ctx:
            ctx.upload_geometry(one.vertices, one.indices, one.blas)
            ctx.reserve_scene(8, 8)
            ctx.set_config(cfg)
            for s in (first, three):
                ctx.upload_scene(s.objects, s.tlas, s.lights, s.instances)
                check(ctx, rays_through(-6, 6, 20_000, 6), len(s.instances))
                ctx.render_frame(_lib.MODE_WAVEFRONT_PRECISION)
            images.append(ctx.read_image(_lib.IMAGE_ACCUM))
    assert np.array_equal(images[0], images[1])
