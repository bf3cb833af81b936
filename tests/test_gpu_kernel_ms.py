"""ae_last_kernel_ms where a call does more than one launch: a frame that builds
structures first reports its kernels alone, and a batch in chunks all of its
kernels.  Times are compared with bounds far from either side: the build takes
longer than the kernel of a one-pixel frame, and a batch of many chunks longer
than its last chunk."""
import ctypes

import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes
from test_gpu_exact import field

pytestmark = pytest.mark.gpu
L = _lib


def kernel_ms(ctx):
    ms = ctypes.c_float()
    L.check(L.lib().ae_last_kernel_ms(ctx.handle, ctypes.byref(ms)), ctx.handle)
    return ms.value


@pytest.mark.parametrize("mode", [L.MODE_COMPUTE_ONLY, L.MODE_DEFERRED])
def test_frame_that_builds(mode):
    s = field()
    with Context(64, 48, hybrid=True) as ctx:
        # A kernel's first launch in a process loads its code.
        ctx.upload(s)
        ctx.prepare_fast()
        ctx.build_gbuffer()
        ctx.render_frame(mode)
        assert ctx.plain_walk_used()
    with Context(640, 480, hybrid=True) as ctx:
        ctx.upload(s)
        cfg = ctx.get_config().copy()
        cfg["depth"] = 1
        ctx.set_config(cfg)
        if mode == L.MODE_DEFERRED:
            ctx.set_plain_walk(L.PLAIN_WALK_REFERENCE)
            ctx.build_gbuffer()
            ctx.set_plain_walk(L.PLAIN_WALK_AUTO)
        times, used = [], []
        for _ in range(12):
            ctx.render_frame(mode)
            L.check(L.lib().ae_synchronize(ctx.handle), ctx.handle)
            used.append(ctx.plain_walk_used())
            times.append(kernel_ms(ctx))
        assert not used[0] and used[-1]
        build = used.index(True)
        # The structures' build takes over 1.5 ms here, the kernel well under 1.
        assert times[build] < 1.5 * max(times[build + 1:]) + 0.3, times


def test_batch_in_chunks():
    s = scenes.instanced_meshes(levels=(4, 3, 3, 2, 2), grid=64, n_instances=80)
    rng = np.random.default_rng(2)
    n = 1_500_000
    rays = np.zeros(n, L.RAY)
    o, d = rng.uniform(0, 100, (n, 3)), rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    for k, x in enumerate("xyz"):
        rays["o" + x], rays["d" + x] = o[:, k], d[:, k]
    rays["tnear"] = 0.001
    tmax = np.full(n, 200.0, np.float32)
    with Context(64, 48) as ctx:
        ctx.upload(s)
        ctx.set_plain_walk(L.PLAIN_WALK_REFERENCE)
        for _ in range(2):
            ctx.any_hit(rays[:65536], tmax[:65536])
            small = kernel_ms(ctx)
            ctx.any_hit(rays, tmax)
            whole = kernel_ms(ctx)
        assert 0 < small and whole > 4 * small, (small, whole)
        ctx.render_frame(L.MODE_COMPUTE_ONLY)
        assert 0 < kernel_ms(ctx) != whole
