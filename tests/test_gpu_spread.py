"""Small ray batches put fewer rays in each warp: every count at the edges of
that rule (one ray, a warp, a block, the counts where the number of lanes per
warp changes, the first count with full warps) gives the reference walk's hits
bit for bit (tolerance zero)."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def traced():
    s = scenes.instanced_meshes(width=64, height=48, levels=(4, 3, 3, 2, 2), grid=64, n_instances=80)
    ctx = Context(64, 48)
    ctx.upload(s)
    rng = np.random.default_rng(12)
    n = 60_000
    rays = np.zeros(n, _lib.RAY)
    o, d = rng.uniform(0, 100, (n, 3)), rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    for k, x in enumerate("xyz"):
        rays["o" + x], rays["d" + x] = o[:, k], d[:, k]
    rays["tnear"] = 0.001
    yield ctx, rays, {v: ctx.closest_hit(rays, v) for v in (_lib.VARIANT_PLAIN, _lib.VARIANT_PLAIN_WT)}
    ctx.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 129, 2072, 2073, 2368, 2369, 4096, 4097, 4737, 33152, 33153, 37888, 37889, 60000])
def test_small_batches(traced, n):
    ctx, rays, want = traced
    for v, w in ((_lib.VARIANT_FAST, _lib.VARIANT_PLAIN), (_lib.VARIANT_FAST_WALK, _lib.VARIANT_PLAIN),
                 (_lib.VARIANT_QUANT, _lib.VARIANT_PLAIN_WT)):
        got = ctx.closest_hit(rays[:n], v)
        assert np.array_equal(got.view(np.uint8), want[w][:n].view(np.uint8)), (n, v)
