"""Two-level traversal where many instances overlap: a ray enters one after the other and takes the rest of a node's
instances off the stack between them. Stage entry points with opaque and non-opaque materials on both sides of the limit
of the kernel with eight lanes per ray, and frames on both sides of the chunk size (1,000,000 paths) from which queues of
any length are traced with a lane per ray."""
import numpy as np
import pytest

from conftest import assert_bits_equal, random_rays

pytestmark = pytest.mark.gpu


def crowd(bsm, opaque, w=64, h=48):
    """Instances scaled up so that a ray crosses dozens of their boxes."""
    sc = bsm.generate_instanced_scene(seed=9, instances=400, width=w, height=h, sphere_res=8, ground=8)
    xf = sc.inst_transform.reshape(-1, 3, 4)
    xf[1:, :, :3] *= 4.0
    sc.inst_transform = xf.reshape(sc.inst_transform.shape)
    if not opaque:
        sc.materials[::2, 5], sc.materials[::2, 6] = 0.7, bsm.BSM_BLEND_TRANSLUCENT
        sc.materials[1::4, 5], sc.materials[1::4, 6] = 0.0, bsm.BSM_BLEND_ALPHA_TEST
    return sc


@pytest.mark.parametrize("n", [1, 37, 12161, 60000, 60001])
@pytest.mark.parametrize("opaque", [True, False])
def test_stage_entry_points_through_overlapping_instances(bsm, ctx, oracle, n, opaque):
    sc = crowd(bsm, opaque)
    sid, osc = ctx.load_instanced(sc), oracle.OracleScene(sc)
    rays = random_rays(n, -1.5, 1.5, seed=n)
    assert np.array_equal(ctx.trace_closest(sid, rays), osc.trace(rays))
    assert np.array_equal(ctx.trace_any(sid, rays) != 0, osc.trace(rays, any_hit=True)[:, 1] != 0xFFFFFFFF)
    ctx.release(sid)


@pytest.mark.parametrize("w,h", [(300, 200), (1000, 1000), (1001, 1000)])
@pytest.mark.parametrize("opaque", [True, False])
def test_frames_of_overlapping_instances(bsm, ctx, oracle, w, h, opaque):
    sc = crowd(bsm, opaque, w, h)
    sid = ctx.load_instanced(sc)
    det = bsm.BSM_PT_DETERMINISTIC
    imgs, st = ctx.render(sid, [sc.camera], bsm.settings(spp=1, max_segments=3, seed=8, flags=det))
    ref, ost, _ = oracle.OracleScene(sc).render(sc.camera.as_array(), spp=1, max_segments=3, seed=8, flags=det)
    assert list(st.rays_per_segment[:3]) == [int(x) for x in ost[:3]]
    assert_bits_equal(imgs[0][..., :3], ref[..., :3])
    ctx.release(sid)
