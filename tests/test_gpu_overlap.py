"""The wavefront form's shadow stages of neighbouring bounces run beside one
another and beside the next extend.  Frames equal the plain megakernel's bit
for bit (tolerance zero) where a wrong order would show: depths below, at and
above the number of shadow sets, several samples a frame, accumulated frames,
and a context that got memory for one set only."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu


def accumulate(s, mode, depth, samples, fail_after=None):
    cfg = s.config.copy()
    cfg["depth"], cfg["samples"] = depth, samples
    with Context(int(cfg["width"]), int(cfg["height"]), samples=samples) as ctx:
        ctx.upload(s)
        if fail_after is not None:
            ctx.prepare_fast()
            _lib.lib().ae_debug_fail_alloc_after(fail_after)
        try:
            for b in range(3):
                cfg["batch"] = b
                ctx.set_config(cfg)
                ctx.render_frame(mode)
        finally:
            _lib.lib().ae_debug_fail_alloc_after(-1)
        return ctx.read_image(_lib.IMAGE_ACCUM).view(np.uint32)


@pytest.mark.parametrize("depth,samples", [(1, 1), (2, 2), (3, 1), (4, 3), (9, 1)])
def test_overlapped_stages(depth, samples):
    s = scenes.hybrid_box(width=131, height=77, depth=6)
    want = accumulate(s, _lib.MODE_COMPUTE_ONLY, depth, samples)
    assert np.array_equal(accumulate(s, _lib.MODE_WAVEFRONT, depth, samples), want)


# The context's eleventh array or a later one (shadow entries) does not fit twice.
@pytest.mark.parametrize("fail_after", [9, 11, 15, 17])
def test_one_set(fail_after):
    s = scenes.hybrid_box(width=131, height=77, depth=6)
    want = accumulate(s, _lib.MODE_COMPUTE_ONLY, 5, 1)
    assert np.array_equal(accumulate(s, _lib.MODE_WAVEFRONT, 5, 1, fail_after), want)
