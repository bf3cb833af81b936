"""The wavefront form's second set of light samples is held for speed alone: an
allocation that fails after it was taken gives it back and is tried again, so
what one set left room for still runs.  Frames and answers are the same
(tolerance zero)."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu
L = _lib


def steps(ctx, rays, tmax):
    """The calls that allocate for the first time after a wavefront frame."""
    cfg = ctx.get_config().copy()
    cfg["batch"] = 0

    def precision():
        ctx.render_frame(L.MODE_WAVEFRONT_PRECISION)
        return ctx.read_image(L.IMAGE_ACCUM)

    def hybrid():
        ctx.build_gbuffer()
        ctx.render_frame(L.MODE_DEFERRED)
        return ctx.read_deferred_accum()

    def reduced():
        low = cfg.copy()
        low["traceScale"] = 0.75
        ctx.set_config(low)
        ctx.render_frame(L.MODE_DEFERRED)
        ctx.set_config(cfg)
        return ctx.read_image(L.IMAGE_DISPLAY)

    return {"precision": precision, "hybrid": hybrid, "reduced": reduced,
            "any hit": lambda: ctx.any_hit(rays, tmax),
            "closest hit": lambda: ctx.closest_hit(rays, L.VARIANT_PLAIN)}


@pytest.mark.parametrize("call", ["precision", "hybrid", "reduced", "any hit", "closest hit"])
def test_allocation_after_the_queues(call):
    s = scenes.hybrid_box(width=131, height=77, depth=6)
    rng = np.random.default_rng(1)
    rays = np.zeros(5000, L.RAY)
    for x in "xyz":
        rays["o" + x], rays["d" + x] = rng.uniform(1, 9, len(rays)), rng.normal(size=len(rays))
    rays["tnear"] = 0.001
    tmax = np.full(len(rays), 3.0, np.float32)

    def run(fail_after):
        with Context(131, 77, hybrid=True) as ctx:
            ctx.upload(s)
            if call == "reduced":
                ctx.build_gbuffer()
            ctx.render_frame(L.MODE_WAVEFRONT)
            L.lib().ae_debug_fail_alloc_after(fail_after)
            try:
                got = steps(ctx, rays, tmax)[call]()
            finally:
                left = L.lib().ae_debug_fail_alloc_after(-1)
            assert left == 0
            # And the wavefront form goes on, on one set.
            ctx.render_frame(L.MODE_WAVEFRONT)
            return got, ctx.read_image(L.IMAGE_ACCUM)

    want = run(-1)
    for k in range({"precision": 4, "hybrid": 8, "reduced": 1, "any hit": 3, "closest hit": 2}[call]):
        got = run(k)
        assert np.array_equal(got[0].view(np.uint8), want[0].view(np.uint8)), k
        assert np.array_equal(got[1].view(np.uint8), want[1].view(np.uint8)), k


def test_hybrid_images_after_a_failed_allocation():
    """A failed allocation of the hybrid images is an error of that call; the
    next one allocates what is missing."""
    s = scenes.hybrid_box(width=131, height=77, depth=3)

    def frame(ctx):
        ctx.build_gbuffer()
        ctx.render_frame(L.MODE_DEFERRED)
        return ctx.read_deferred_accum()

    with Context(131, 77, hybrid=True) as ctx:
        ctx.upload(s)
        want = frame(ctx)
    for k in range(8):
        with Context(131, 77, hybrid=True) as ctx:
            ctx.upload(s)
            L.lib().ae_debug_fail_alloc_after(k)
            try:
                with pytest.raises(L.AeError):
                    frame(ctx)
            finally:
                L.lib().ae_debug_fail_alloc_after(-1)
            assert np.array_equal(frame(ctx), want), k
