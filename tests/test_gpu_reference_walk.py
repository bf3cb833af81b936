"""The wavefront forms against the plain megakernel held on the reference walk
(ae_set_plain_walk), so that neither side uses the structures under test: the
same frames bit for bit (tolerance zero), and the counterpart for frames that
trace enough rays for the plain form to build in between."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes
from test_gpu_exact import boxes, field

pytestmark = pytest.mark.gpu
L = _lib


def accumulate(s, mode, walk, width, height, frames, depth):
    with Context(width, height) as ctx:
        ctx.upload(s)
        ctx.set_plain_walk(walk)
        cfg = ctx.get_config().copy()
        cfg["depth"] = depth
        for k in range(frames):
            cfg["batch"] = k
            ctx.set_config(cfg)
            ctx.render_frame(mode)
            assert mode != L.MODE_COMPUTE_ONLY or walk == L.PLAIN_WALK_AUTO or not ctx.plain_walk_used()
        return ctx.read_image(L.IMAGE_ACCUM).view(np.uint8), ctx.read_image(L.IMAGE_DISPLAY)


@pytest.mark.parametrize("scene,width,height", [(scenes.hybrid_box, 480, 270), (scenes.textured_box, 320, 240),
                                                (lambda: field(True), 320, 180), (boxes, 320, 180)])
def test_wavefront_against_the_reference_walk(scene, width, height):
    s = scene()
    want = accumulate(s, L.MODE_COMPUTE_ONLY, L.PLAIN_WALK_REFERENCE, width, height, 3, 6)
    for mode, walk in ((L.MODE_WAVEFRONT, L.PLAIN_WALK_AUTO), (L.MODE_COMPUTE_ONLY, L.PLAIN_WALK_AUTO)):
        got = accumulate(s, mode, walk, width, height, 3, 6)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), mode
