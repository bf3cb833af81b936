"""ae_set_plain_walk: which walk the plain forms take, when a call may build
the structures, and that frames do not depend on either (bit for bit,
tolerance zero)."""
import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes
from test_gpu_exact import boxes, field

pytestmark = pytest.mark.gpu
L = _lib


def frames(s, n, mode, prepare=False, width=96, height=64, samples=1, **settings):
    """n accumulated compute-only frames: (images after each, which walk)."""
    images, used = [], []
    with Context(width, height, samples=samples) as ctx:
        ctx.upload(s)
        ctx.set_plain_walk(mode)
        if prepare:
            ctx.prepare_fast()
        cfg = ctx.get_config().copy()
        cfg["samples"] = samples
        for k, v in settings.items():
            cfg[k] = v
        for k in range(n):
            cfg["batch"] = k
            ctx.set_config(cfg)
            ctx.render_frame(L.MODE_COMPUTE_ONLY)
            used.append(ctx.plain_walk_used())
            images.append((ctx.read_image(L.IMAGE_ACCUM).view(np.uint8), ctx.read_image(L.IMAGE_DISPLAY)))
    return images, used


def same(a, b):
    return all(np.array_equal(x, y) for p, q in zip(a, b) for x, y in zip(p, q))


@pytest.mark.parametrize("scene", [field, boxes, scenes.cornell_box, scenes.textured_box, scenes.hybrid_box,
                                   lambda: scenes.instanced_meshes(levels=(4, 3, 3, 2, 2), grid=64, n_instances=80)])
def test_prepared_structures_are_used(scene):
    """Scenes within the exact walks' premises, textured ones among them, trace
    on prepared structures, after a refit too, and render the reference walk's
    frames."""
    s = scene()
    want, used = frames(s, 3, L.PLAIN_WALK_REFERENCE, prepare=True, depth=5)
    assert not any(used)
    got, used = frames(s, 3, L.PLAIN_WALK_PREPARED, prepare=True, depth=5)
    assert all(used)
    assert same(got, want)
    if len(s.instances) < 2:
        return
    rng = np.random.default_rng(1)
    with Context(96, 64) as ctx:
        ctx.upload(s)
        ctx.prepare_fast()
        pose = s.instances
        for _ in range(3):
            pose = scenes.random_walk(pose, rng)
            ctx.refit_instances(pose)
            ctx.prepare_fast()
            ctx.render_frame(L.MODE_COMPUTE_ONLY)
            assert ctx.plain_walk_used()


def moving_sphere():
    s = scenes.hybrid_box()
    ball = np.flatnonzero(s.objects["shapeType"] == L.SHAPE_SPHERE)[0]
    s.objects["x2"][ball] += np.float32(0.5)
    return s


@pytest.mark.parametrize("scene", [scenes.media_box, moving_sphere])
def test_scenes_for_the_reference_walk(scene):
    """Media and spheres that move within a frame keep the reference walk,
    however many rays are traced."""
    s = scene()
    want, _ = frames(s, 3, L.PLAIN_WALK_REFERENCE, width=320, height=240, samples=16, depth=3)
    got, used = frames(s, 3, L.PLAIN_WALK_AUTO, width=320, height=240, samples=16, depth=3)
    assert not any(used)
    assert same(got, want)


@pytest.mark.parametrize("scene,width,height,samples", [(field, 160, 120, 2), (boxes, 320, 240, 16)])
def test_build_in_mid_sequence(scene, width, height, samples):
    """Frames before and after the call that builds."""
    s = scene()
    want, _ = frames(s, 6, L.PLAIN_WALK_REFERENCE, width=width, height=height, samples=samples, depth=5)
    got, used = frames(s, 6, L.PLAIN_WALK_AUTO, width=width, height=height, samples=samples, depth=5)
    assert not used[0] and used[-1] and used == sorted(used)
    assert same(got, want)


def test_prepared_mode_builds_nothing():
    s = field()
    rays = np.zeros(2_000_000, L.RAY)
    rays["dx"], rays["tnear"] = 1.0, 0.001
    with Context(320, 240) as ctx:
        ctx.upload(s)
        ctx.set_plain_walk(L.PLAIN_WALK_PREPARED)
        cfg = ctx.get_config().copy()
        cfg["samples"] = 64
        ctx.set_config(cfg)
        ctx.render_frame(L.MODE_COMPUTE_ONLY)
        live = L.lib().ae_debug_live_allocations()
        ctx.render_frame(L.MODE_COMPUTE_ONLY)
        assert not ctx.plain_walk_used() and L.lib().ae_debug_live_allocations() == live
        ctx.any_hit(rays, np.ones(len(rays), np.float32))
        assert not ctx.plain_walk_used()
        ctx.prepare_fast()
        ctx.render_frame(L.MODE_COMPUTE_ONLY)
        assert ctx.plain_walk_used()
        with pytest.raises(L.AeError):
            ctx.set_plain_walk(3)


def test_prepared_after_a_failed_build():
    """A build that fails leaves its call to the reference walk and is not tried
    again by itself; structures that the caller then prepares are used."""
    s = field()
    want, _ = frames(s, 3, L.PLAIN_WALK_REFERENCE, width=160, height=120, samples=2, depth=5)
    with Context(160, 120, samples=2) as ctx:
        ctx.upload(s)
        cfg = ctx.get_config().copy()
        cfg["samples"], cfg["depth"] = 2, 5
        got, used = [], []
        ctx.set_config(cfg)
        ctx.render_frame(L.MODE_COMPUTE_ONLY)
        # Pending until a call allocates, which is the one that builds.
        L.lib().ae_debug_fail_alloc_after(0)
        try:
            for _ in range(30):
                ctx.render_frame(L.MODE_COMPUTE_ONLY)
                assert not ctx.plain_walk_used()
        finally:
            L.lib().ae_debug_fail_alloc_after(-1)
        ctx.prepare_fast()
        for k in range(3):
            cfg["batch"] = k
            ctx.set_config(cfg)
            ctx.render_frame(L.MODE_COMPUTE_ONLY)
            used.append(ctx.plain_walk_used())
            got.append((ctx.read_image(L.IMAGE_ACCUM).view(np.uint8), ctx.read_image(L.IMAGE_DISPLAY)))
    assert all(used)
    assert same(got, want)


def test_capture():
    """A compute-only frame recorded into a caller's graph on the context's
    stream, at the call that would build: it is recorded on the reference walk
    and builds nothing."""
    import torch
    s = field()
    with Context(96, 64) as ref:
        ref.upload(s)
        ref.set_plain_walk(L.PLAIN_WALK_REFERENCE)
        ref.render_frame(L.MODE_COMPUTE_ONLY)
        want = ref.read_image(L.IMAGE_ACCUM).view(np.uint8)
    with Context(96, 64) as ctx:
        ctx.upload(s)
        cfg = ctx.get_config().copy()
        cfg["samples"] = 1024  # more rays than any build costs
        ctx.set_config(cfg)
        stream = torch.cuda.ExternalStream(L.lib().ae_stream(ctx.handle))
        live = L.lib().ae_debug_live_allocations()
        heavy, light = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(heavy, stream=stream, capture_error_mode="thread_local"):
            ctx.render_frame(L.MODE_COMPUTE_ONLY)
        assert not ctx.plain_walk_used() and L.lib().ae_debug_live_allocations() == live
        cfg["samples"] = 1
        ctx.set_config(cfg)
        with torch.cuda.graph(light, stream=stream, capture_error_mode="thread_local"):
            ctx.render_frame(L.MODE_COMPUTE_ONLY)
        for _ in range(2):
            with torch.cuda.stream(stream):
                light.replay()
            L.check(L.lib().ae_synchronize(ctx.handle), ctx.handle)
            assert np.array_equal(ctx.read_image(L.IMAGE_ACCUM).view(np.uint8), want)
        # Outside a capture the same call builds.
        cfg["samples"] = 1024
        cfg["depth"] = 1
        ctx.set_config(cfg)
        ctx.render_frame(L.MODE_COMPUTE_ONLY)
        assert ctx.plain_walk_used()
        del heavy, light


def test_display_only_frames_trace_nothing():
    """Grading an image again builds no structures, however large the image,
    and does not count towards the build of a later frame."""
    s = field()
    with Context(1024, 1024) as ctx:
        ctx.upload(s)
        cfg = ctx.get_config().copy()
        cfg["samples"], cfg["displayOnly"] = 8, 1
        ctx.set_config(cfg)
        live = L.lib().ae_debug_live_allocations()
        for _ in range(4):
            ctx.render_frame(L.MODE_COMPUTE_ONLY)
        assert L.lib().ae_debug_live_allocations() == live and not ctx.plain_walk_used()
        rays = np.zeros(64, L.RAY)
        rays["dx"], rays["tnear"] = 1.0, 0.001
        ctx.any_hit(rays, np.ones(64, np.float32))
        assert not ctx.plain_walk_used()


def test_small_scenes_stay_on_the_reference_walk():
    """Any hit and the hybrid passes of a handful of objects, prepared or not;
    PREPARED still takes the structures there."""
    s = scenes.cornell_box()
    rng = np.random.default_rng(3)
    rays = np.zeros(300_000, L.RAY)
    for x in "xyz":
        rays["o" + x], rays["d" + x] = rng.uniform(1, 9, len(rays)), rng.normal(size=len(rays))
    rays["tnear"] = 0.001
    tmax = np.full(len(rays), 3.0, np.float32)
    got = {}
    for mode in (L.PLAIN_WALK_AUTO, L.PLAIN_WALK_PREPARED, L.PLAIN_WALK_REFERENCE):
        with Context(96, 64, hybrid=True) as ctx:
            ctx.upload(s)
            ctx.prepare_fast()
            ctx.set_plain_walk(mode)
            got[mode] = ctx.any_hit(rays, tmax)
            used = [ctx.plain_walk_used()]
            ctx.build_gbuffer()
            used.append(ctx.plain_walk_used())
            ctx.render_frame(L.MODE_DEFERRED)
            used.append(ctx.plain_walk_used())
            assert used == [mode == L.PLAIN_WALK_PREPARED] * 3
    assert all(np.array_equal(g, got[L.PLAIN_WALK_REFERENCE]) for g in got.values())


def test_builds_when_it_pays():
    """The first calls on new scenes: a large scene's compute-only frames build
    at once or nearly, a small one's only after a score of frames, a few any-hit
    rays never."""
    big = scenes.wavefront_scene(seed=3, width=480, height=270, depth=8, n_meshes=8, n_instances=64, n_lights=4,
                                 target_tris=60_000)
    for s, w, h, first, last in ((big, 480, 270, 0, 1), (scenes.cornell_box(), 320, 240, 12, 40)):
        with Context(w, h) as ctx:
            ctx.upload(s)
            used = []
            for _ in range(last + 1):
                ctx.render_frame(L.MODE_COMPUTE_ONLY)
                used.append(ctx.plain_walk_used())
            assert True in used and first <= used.index(True)
    with Context(64, 48) as ctx:
        ctx.upload(big)
        rays = np.zeros(10_000, L.RAY)
        rays["dx"], rays["tnear"] = 1.0, 0.001
        for _ in range(5):
            ctx.any_hit(rays, np.ones(len(rays), np.float32))
            assert not ctx.plain_walk_used()
