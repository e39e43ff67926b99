"""Chunks of over 3,000,000 paths trace the shadow rays of the camera rays' hits towards the lights in a launch of
their own: frames on both sides of the limit against the oracle, with one light and with two, with and without
non-opaque materials, and with the stages timed one by one."""
import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1000, 1000), (1001, 1000)])   # x 3 samples: the limit, and over it
@pytest.mark.parametrize("lights", [1, 2])
@pytest.mark.parametrize("opaque", [True, False])
def test_both_sides_of_the_limit(bsm, ctx, oracle, w, h, lights, opaque):
    sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=21, width=w, height=h)
    if lights == 2:
        sc.lights = np.concatenate([sc.lights, np.array([[0.5, 0.2, 0.84, 0.6, 0.5, 0.4]], np.float32)])
    if not opaque:
        sc.materials[1::2, 5], sc.materials[1::2, 6] = 0.6, bsm.BSM_BLEND_TRANSLUCENT
    sid = ctx.load_scene(sc)
    det = bsm.BSM_PT_DETERMINISTIC
    ref, ost, _ = oracle.OracleScene(sc).render(sc.camera.as_array(), spp=3, max_segments=2, seed=5, flags=det)
    for flags in (det, det | bsm.BSM_PT_STAGE_TIMING):
        imgs, st = ctx.render(sid, [sc.camera], bsm.settings(spp=3, max_segments=2, seed=5, flags=flags))
        assert list(st.rays_per_segment[:2]) == [int(x) for x in ost[:2]]
        assert_bits_equal(imgs[0][..., :3], ref[..., :3])
    ctx.release(sid)
