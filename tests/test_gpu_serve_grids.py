"""A chunk's traversal takes half of the persistent grid when as much work runs or waits beside it, and all of it when it
is most of the work: a request of several chunks, long enough for the kernels with a lane per ray, has the same bits alone,
beside as much other work, beside little, and as rendered by itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_level", [False, True])
@pytest.mark.parametrize("chunk_paths", [0, 300000])
def test_same_bits_with_half_and_whole_grids(bsm, two_level, chunk_paths):
    with bsm.Context(0) as ctx:
        if two_level:
            sc = bsm.generate_instanced_scene(seed=6, instances=120, sphere_res=8, ground=16)
            sid = ctx.load_instanced(sc)
        else:
            sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=12)
            sid = ctx.load_scene(sc)
        other = ctx.load_scene(bsm.generate_scene(bsm.BSM_SCENE_TERRAIN, seed=2, grid=64, spheres=40))

        def cam(w, h):
            return bsm.make_camera(tuple(sc.camera.position), tuple(sc.camera.front), width=w, height=h)

        big = (sid, cam(480, 360), 5, 4, 77)   # 864,000 paths
        ref, _ = ctx.render(sid, [big[1]], bsm.settings(spp=5, max_segments=4, seed=77, flags=bsm.BSM_PT_DETERMINISTIC))
        ctx.server_start(deterministic=True, chunk_paths=chunk_paths)
        try:
            images = []
            for beside in ([], [(other, cam(512, 400), 5, 8, k) for k in range(3)], [(other, cam(64, 48), 1, 2, 5)]):
                reqs = [ctx.submit(*big)] + [ctx.submit(*r) for r in beside]
                for rid, _ in reqs:
                    ctx.wait(rid)
                images.append(reqs[0][1].copy())
        finally:
            ctx.server_stop()
    for img in images:
        assert np.array_equal(img[..., :3].view(np.uint32), ref[0][..., :3].view(np.uint32))
