"""Rays that start at about tnear from a surface that is a face of its mesh's
boxes: the walks' boxes may not end before the surface does.  The triangle
test decides whether a hit counts as beyond tnear, so an optimised walk may
report such a hit where the reference walk's boxes end a rounding earlier,
but it never loses one (tolerance zero)."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu


def room(size, at):
    """A floor, a ceiling and a sphere between in one mesh of `size` units."""
    lib = scenes.MeshLibrary()
    v, i = scenes.quad_mesh((0, 0, size), (size, 0, 0))
    top, ball = v.copy(), scenes.icosphere(3, 0.1 * size)
    top["py"] += size
    b = ball[0].copy()
    b["py"] += 0.5 * size
    h = lib.add(np.concatenate([v, top, b]), np.concatenate([i, i + 4, ball[1] + 8]).astype(np.uint32))
    e = scenes.entity(_lib.SHAPE_MESH, _lib.MAT_LAMBERTIAN, (at, at, at), mesh=h)
    return scenes._finish([e], lib, scenes.make_config(64, 48, (0, 0, 20), (0, 0, 0)), "room")


@pytest.mark.parametrize("size,at", [(100.0, 0.0), (100.0, 37.3), (1000.0, 0.0), (10.0, 3.1), (0.5, 0.1)])
@pytest.mark.parametrize("side", [0.0, 1.0])
@pytest.mark.parametrize("tnear", [0.001, 0.0])
def test_hits_at_tnear(size, at, side, tnear):
    rng = np.random.default_rng(7)
    n = 200_000
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:, 1] = np.abs(d[:, 1]) * (1.0 if side else -1.0)
    t = 0.001 + rng.uniform(-1, 1, n) * rng.choice([1e-7, 1e-6, 1e-5, 1e-4], n) * size / 100
    hit = np.stack([rng.uniform(-0.5, 0.5, n) * size, np.full(n, side * size), rng.uniform(-0.5, 0.5, n) * size], 1)
    o = hit + at - d * t[:, None]
    rays = np.zeros(n, _lib.RAY)
    for k, x in enumerate("xyz"):
        rays["o" + x], rays["d" + x] = o[:, k], d[:, k]
    rays["tnear"] = tnear
    with Context(64, 48) as ctx:
        ctx.upload(room(size, at))
        for plain, fast in ((_lib.VARIANT_PLAIN, (_lib.VARIANT_FAST, _lib.VARIANT_FAST_WALK)),
                            (_lib.VARIANT_PLAIN_WT, (_lib.VARIANT_QUANT,))):
            want = ctx.closest_hit(rays, plain)
            far = np.where(want["object"] == _lib.MISS, np.inf, want["t"])
            for v in fast:
                # The whole batch, and a part of it that four lanes a ray walk.
                for m in (n, 5000):
                    got = ctx.closest_hit(rays[:m], v)
                    assert (np.where(got["object"] == _lib.MISS, np.inf, got["t"]) <= far[:m]).all(), (v, m)
