"""Instances that move (ae_refit_instances): trees small enough for the
one-block level passes and trees with a launch per level, several moves, and a
wavefront frame whose captured graph outlives them.  Hits and frames must be
those of a context that was given the moved scene outright; the optimised
hits the reference walk's (tolerance zero)."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu


def crowd(n, seed):
    rng = np.random.default_rng(seed)
    lib = scenes.MeshLibrary()
    hs = [lib.add(*scenes.icosphere(1, 0.4)), lib.add(*scenes.box_mesh((0.3, 0.5, 0.4)))]
    side = max(4.0, n ** (1 / 3) * 1.5)
    ents = [scenes.entity(_lib.SHAPE_QUAD, _lib.MAT_DIFFUSE_LIGHT, (0, 2 * side, 0), emission=20.0, u=(side, 0, 0),
                          v=(0, 0, side))]
    for k in range(n):
        ents.append(scenes.entity(_lib.SHAPE_MESH, _lib.MAT_LAMBERTIAN, rng.uniform(0, side, 3), mesh=hs[k % 2],
                                  rotation=scenes.random_quat(rng), scale=float(rng.uniform(0.5, 2.0)),
                                  albedo=tuple(float(x) for x in rng.uniform(0.2, 0.8, 3))))
    cfg = scenes.make_config(64, 48, (side / 2, side, 3 * side), (side / 2, side / 2, side / 2), depth=3, sky=(0.2, 0.3, 0.4))
    return scenes._finish(ents, lib, cfg, "crowd"), side


@pytest.mark.parametrize("n", [1, 2, 33, 1000, 3500, 4200])
def test_moves(n):
    s, side = crowd(n, n)
    rng = np.random.default_rng(n + 1)
    rays = np.zeros(20_000, _lib.RAY)
    o, d = rng.uniform(0, side, (len(rays), 3)), rng.normal(size=(len(rays), 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    for k, x in enumerate("xyz"):
        rays["o" + x], rays["d" + x] = o[:, k], d[:, k]
    rays["tnear"] = 0.001
    at = s.instances
    with Context(64, 48) as ctx:
        ctx.upload(s)
        for move in range(3):
            if move:
                at = scenes.random_walk(at, rng, step=0.3, angle=0.5)
                ctx.refit_instances(at)
            plain = ctx.closest_hit(rays, _lib.VARIANT_PLAIN)
            for v in (_lib.VARIANT_FAST, _lib.VARIANT_FAST_WALK):
                assert np.array_equal(ctx.closest_hit(rays, v).view(np.uint8), plain.view(np.uint8)), (move, v)
            ctx.render_frame(_lib.MODE_WAVEFRONT)
            frame = ctx.read_image(_lib.IMAGE_FRAME)
            objects, tlas, instances = ctx.download_scene()
            with Context(64, 48) as other:
                other.upload_geometry(s.vertices, s.indices, s.blas)
                other.upload_scene(objects, tlas, s.lights, instances)
                other.set_config(ctx.get_config())
                assert np.array_equal(other.closest_hit(rays, _lib.VARIANT_PLAIN).view(np.uint8), plain.view(np.uint8))
                other.render_frame(_lib.MODE_WAVEFRONT)
                assert np.array_equal(other.read_image(_lib.IMAGE_FRAME), frame), move
            assert np.array_equal(instances.view(np.uint8), at.view(np.uint8))
            old = [float(x) for x in objects["prevRotX"][objects["shapeType"] == _lib.SHAPE_MESH][:3]]
            assert all(np.isfinite(old))
