"""Geometry uploaded again under an uploaded scene: structures are built from
it only when the scene's meshes lie in it."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu
L = _lib


def test_geometry_after_the_scene():
    s = scenes.cornell_box(width=64, height=48)
    small = scenes.MeshLibrary()
    small.add(*scenes.quad_mesh((0, 0, 1), (1, 0, 0)))
    v, i, b = small.arrays()
    moved = s.vertices.copy()
    moved["py"] *= np.float32(0.75)
    with Context(64, 48) as ctx:
        ctx.upload(s)
        rays = ctx.camera_rays()
        before = ctx.closest_hit(rays, L.VARIANT_FAST)
        # Too short for the scene's instances: refused, and nothing is read.
        ctx.upload_geometry(v, i, b)
        for call in (ctx.prepare_fast, lambda: ctx.closest_hit(rays, L.VARIANT_FAST),
                     lambda: ctx.render_frame(L.MODE_WAVEFRONT)):
            with pytest.raises(L.AeError) as e:
                call()
            assert e.value.code == -4
        # Part of the scene's instances fit.
        ctx.upload_geometry(s.vertices, s.indices[:12], s.blas)
        for _ in range(2):
            with pytest.raises(L.AeError):
                ctx.prepare_fast()
        # The same layout with other vertices is what the scene now shows.
        ctx.upload_geometry(moved, s.indices, s.blas)
        got = ctx.closest_hit(rays, L.VARIANT_FAST)
        assert not np.array_equal(got["t"], before["t"])
        ctx.upload_geometry(s.vertices, s.indices, s.blas)
        assert np.array_equal(ctx.closest_hit(rays, L.VARIANT_FAST).view(np.uint8), before.view(np.uint8))
