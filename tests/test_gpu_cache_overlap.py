"""A cached frame traces its training paths beside its render; frames whose stages are timed, and frames of several
chunks, train first. The two orders give the same frames and weights bit for bit (with BSM_PT_DETERMINISTIC every sum
that the order of launches could change is exact; the reported loss alone is summed by atomics, in any order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(bsm):
    return bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=41, spheres=24)


def frames(bsm, ctx, scene, w, h, flags=0, capacity=0, ema=0.0, accumulate=0, n=3):
    sid = ctx.load_scene(scene)
    cam = bsm.make_camera(tuple(scene.camera.position), tuple(scene.camera.front), width=w, height=h)
    cs = bsm.cache_settings(cache_segment=2, train_paths=3001, train_steps=2, train_batch=4096, ema_decay=ema)
    s = bsm.settings(spp=2, seed=9, flags=bsm.BSM_PT_DETERMINISTIC | flags, wavefront_capacity=capacity)
    c = bsm.RadianceCache(ctx, seed=5)
    try:
        out = []
        for k in range(n):
            s.accumulate = accumulate if k else 0   # the context may hold sums of an earlier frame of this camera
            out.append(c.render(sid, cam, s, cs)[0].view(np.uint32).copy())
        return out, c.weights().view(np.uint32).copy()
    finally:
        c.close()
        ctx.release(sid)


# 64x48x2 = 6,144 paths: one chunk, or six of 1,024 (the last one ends the frame) or two (6,143 and one path)
@pytest.mark.parametrize("kw", [dict(capacity=1024), dict(capacity=6143), dict(capacity=6144), dict(no_graph=True),
                                dict(ema=0.9), dict(accumulate=1)])
def test_overlapped_training_gives_the_frames_of_training_first(bsm, ctx, scene, kw):
    kw = dict(kw)
    flags = bsm.BSM_PT_NO_GRAPH if kw.pop("no_graph", False) else 0
    got, gw = frames(bsm, ctx, scene, 64, 48, flags=flags, **kw)
    ref, rw = frames(bsm, ctx, scene, 64, 48, flags=bsm.BSM_PT_STAGE_TIMING, **{**kw, "capacity": 0})
    assert np.array_equal(gw, rw)
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


def test_a_frame_that_the_render_refuses_has_trained_all_the_same(bsm, ctx, scene):
    sid = ctx.load_scene(scene)
    cam = bsm.make_camera(tuple(scene.camera.position), tuple(scene.camera.front), width=64, height=48)
    cs = bsm.cache_settings(cache_segment=2, train_paths=3001, train_steps=2, train_batch=4096)
    c = bsm.RadianceCache(ctx, seed=5)
    try:
        w0 = c.weights().copy()
        with pytest.raises(bsm.BsmError):
            c.render(sid, cam, bsm.settings(spp=0, seed=9), cs)
        w1 = c.weights().view(np.uint32).copy()
    finally:
        c.close()
        ctx.release(sid)
    assert not np.array_equal(w0.view(np.uint32), w1)
    _, ref = frames(bsm, ctx, scene, 64, 48, n=1)
    assert np.array_equal(w1, ref)
