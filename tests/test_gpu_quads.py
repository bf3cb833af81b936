"""Small batches take four lanes a ray: the hits of the batch that has too many
rays for that, bit for bit (tolerance zero), at the edges of the rule, for
rays that the quads leave to the one-lane walk (huge, infinite and NaN
components) and for analytic shapes, with both triangle tests."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu
N = 40_000  # one lane a ray


def rays_in(lo, hi, seed):
    rng = np.random.default_rng(seed)
    rays = np.zeros(N, _lib.RAY)
    o, d = rng.uniform(lo, hi, (N, 3)), rng.normal(size=(N, 3))
    d[1::7, 0] = 0.0
    d[3::97] *= 1e16
    o[5::101, 1] = 1e16
    d[7::103, 2] = np.inf
    d[11::107] = np.nan
    for k, x in enumerate("xyz"):
        rays["o" + x], rays["d" + x] = o[:, k], d[:, k]
    rays["tnear"] = 0.001
    return rays


@pytest.mark.parametrize("name", ["meshes", "box"])
@pytest.mark.parametrize("variant", [_lib.VARIANT_FAST, _lib.VARIANT_QUANT])
def test_quads_equal_one_lane(name, variant):
    s = (scenes.instanced_meshes(width=64, height=48, levels=(4, 3, 3, 2, 2), grid=64, n_instances=80) if name == "meshes"
         else scenes.hybrid_box(width=64, height=48, depth=3))
    rays = rays_in(0, 100, 3) if name == "meshes" else rays_in(-1, 1, 4)
    with Context(64, 48) as ctx:
        ctx.upload(s)
        want = ctx.closest_hit(rays, variant)
        for n in (1, 3, 9, 2367, 2368, 2369, 18943, 18944, 18945):
            got = ctx.closest_hit(rays[:n], variant)
            assert np.array_equal(got.view(np.uint8), want[:n].view(np.uint8)), n
