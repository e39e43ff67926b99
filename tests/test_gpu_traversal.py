"""The traversal kernels against the oracle where their shortcuts could go wrong: exact zeros on edges and
vertices for every dominant axis and sign of the direction; frames on both sides of the chunk sizes at which the
kernel with eight lanes per ray hands over to both kernels (40,960 paths) and these to the one with a lane per ray
(1,000,000), with and without non-opaque materials, in one level and in two; stage entry points and primary outputs at the sizes where their kernels change."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_bits_equal, random_rays

pytestmark = pytest.mark.gpu


def cube_scene(bsm, n=4):
    """The surface of the cube [-2, 2]^3, n x n squares a side with alternating diagonals and windings."""
    P, idx = [], []
    for axis in range(3):
        for side in (-2.0, 2.0):
            base = len(P)
            for i in range(n + 1):
                for j in range(n + 1):
                    p = [0.0, 0.0, 0.0]
                    p[axis], p[(axis + 1) % 3], p[(axis + 2) % 3] = side, -2.0 + 4.0 * i / n, -2.0 + 4.0 * j / n
                    P.append(p)
            for i in range(n):
                for j in range(n):
                    a, b = base + i * (n + 1) + j, base + (i + 1) * (n + 1) + j
                    quad = [(a, b, b + 1), (a, b + 1, a + 1)] if (i + j) % 2 else [(a, a + 1, b), (b + 1, b, a + 1)]
                    idx += quad
    mats = np.array([[0.5, 0.5, 0.5, 0.5, 0.0]], np.float32)
    lights = np.array([[0.3, 0.4, -1.0, 2.0, 2.0, 2.0]], np.float32)
    cam = bsm.make_camera((0.5, 0.5, -1.0), (0.0, 0.0, 1.0), yfov_deg=40.0, width=16, height=16)
    return bsm.SceneData(np.array(P, np.float32), np.array(idx, np.uint32), np.zeros(len(idx), np.uint32), mats, lights,
                         bsm.BSM_SKY_CONSTANT, (0.3, 0.3, 0.3), None, cam)


def lattice_rays(tmin):
    """From lattice points inside the cube through its vertices, edge midpoints and face centres (every edge
    function there is exactly zero or exact in float32), and along the axes."""
    pts = np.array([[x, y, z] for x in (-1, 0, 0.5) for y in (0, 1, -0.5) for z in (-1, 0, 1)], np.float32)
    half = np.arange(-4, 5, dtype=np.float32) * 0.5
    to = []
    for axis in range(3):
        for side in (-2.0, 2.0):
            for u in half:
                for v in half:
                    p = np.zeros(3, np.float32)
                    p[axis], p[(axis + 1) % 3], p[(axis + 2) % 3] = side, u, v
                    to.append(p)
    to = np.array(to)
    o = np.repeat(pts, len(to), 0)
    d = np.tile(to, (len(pts), 1)) - o
    rays = np.concatenate([o, np.full((len(o), 1), tmin, np.float32), d, np.full((len(o), 1), 4.0, np.float32)], 1)
    axes = np.concatenate([np.eye(3), -np.eye(3)]).astype(np.float32)
    ax = np.concatenate([np.repeat(pts, 6, 0), np.full((len(pts) * 6, 1), tmin, np.float32), np.tile(axes, (len(pts), 1)),
                         np.full((len(pts) * 6, 1), 9.0, np.float32)], 1)
    surface = np.concatenate([to, np.full((len(to), 1), tmin, np.float32), to[::-1] * 0.25 + 0.125,
                              np.full((len(to), 1), 9.0, np.float32)], 1)   # origins on the surface: t = 0 hits
    return np.ascontiguousarray(np.concatenate([rays, ax, surface]), np.float32)


@pytest.mark.parametrize("tmin", [0.0, -0.125])   # the second also takes hits at t = 0, all of which are zeros
def test_exact_zeros_match_the_oracle_bit_for_bit(bsm, ctx, oracle, tmin):
    sc = cube_scene(bsm)
    sid = ctx.load_scene(sc)
    rays = lattice_rays(tmin)
    g, c = ctx.trace_closest(sid, rays), oracle.OracleScene(sc).trace(rays)
    assert (c[:, 1] != 0xFFFFFFFF).sum() > 1000
    bad = np.argwhere(g != c)
    assert bad.size == 0, f"{len(bad)} words differ, first ray {rays[bad[0, 0]].tolist()}: {g[bad[0, 0]]} {c[bad[0, 0]]}"
    ctx.release(sid)


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (9, 3, 1), (256, 160, 1), (257, 160, 1), (128, 96, 9), (250, 250, 16),
                                     (251, 250, 16)])
@pytest.mark.parametrize("opaque", [True, False])
def test_both_sides_of_the_group_kernel_limits(bsm, ctx, oracle, w, h, spp, opaque):
    sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=11, width=w, height=h)
    if not opaque:
        sc.materials[1::2, 5], sc.materials[1::2, 6] = 0.6, bsm.BSM_BLEND_TRANSLUCENT
    sid = ctx.load_scene(sc)
    det = bsm.BSM_PT_DETERMINISTIC
    imgs, st = ctx.render(sid, [sc.camera], bsm.settings(spp=spp, max_segments=4, seed=5, flags=det))
    ref, ost, _ = oracle.OracleScene(sc).render(sc.camera.as_array(), spp=spp, max_segments=4, seed=5, flags=det)
    assert list(st.rays_per_segment[:4]) == [int(x) for x in ost[:4]]
    assert_bits_equal(imgs[0][..., :3], ref[..., :3])
    ctx.release(sid)


@pytest.mark.parametrize("n", [1, 31, 33, 40000, 40001, 300007])   # eight lanes per ray up to 40,000
@pytest.mark.parametrize("opaque", [True, False])
def test_stage_entry_points_at_their_kernels_limits(bsm, ctx, oracle, n, opaque):
    sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=12)
    if not opaque:
        sc.materials[::2, 5], sc.materials[::2, 6] = 0.5, bsm.BSM_BLEND_TRANSLUCENT
    sid, osc = ctx.load_scene(sc), oracle.OracleScene(sc)
    rays = random_rays(n, 0.0, 1.0, seed=n)
    rays[n // 2, 4:7] = 0.0   # one that is not traced
    for _ in range(2):        # the second call starts from the work counter that the first one left
        assert np.array_equal(ctx.trace_closest(sid, rays), osc.trace(rays))
        assert np.array_equal(ctx.trace_any(sid, rays) != 0, osc.trace(rays, any_hit=True)[:, 1] != 0xFFFFFFFF)
    ctx.release(sid)


# a tile is 16 x 8 pixels; up to 24,576 pixels go to the kernel with eight lanes per ray
@pytest.mark.parametrize("w,h", [(1, 1), (17, 9), (192, 128), (193, 128), (8, 5001), (5001, 8)])
@pytest.mark.parametrize("which", ["all", "depth", "normals"])
def test_primary_outputs_at_their_kernels_limits(bsm, ctx, oracle, w, h, which):
    sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=13, width=w, height=h)
    sid, cam = ctx.load_scene(sc), sc.camera
    d0, g0, h0 = oracle.OracleScene(sc).primary(cam.as_array())
    d, g, hp = np.zeros_like(d0), np.zeros_like(g0), np.zeros_like(h0)
    out = bsm.PrimaryOutput()
    if which != "normals":
        out.depth = d.ctypes.data
    for k in range(4):
        if which == "all" or (which == "normals" and k == 1):
            out.gbuffer[k] = g[k].ctypes.data
    if which == "all":
        out.hit_positions = hp.ctypes.data
    out.location = bsm.BSM_HOST
    ctx.check(ctx._L.bsm_render_primary(ctx.h, sid, C.byref(cam), None, 0.0, 0.0, C.byref(out)))
    if which != "normals":
        assert_bits_equal(d, d0)
    if which == "normals":
        assert_bits_equal(g[1], g0[1])
    if which == "all":
        assert_bits_equal(g, g0)
        assert_bits_equal(hp, h0)
    ctx.release(sid)


# eight lanes per ray up to 98,304 paths (512 x 192); beyond, queues of up to 90,000 rays
@pytest.mark.parametrize("w,h", [(1, 1), (13, 7), (512, 192), (513, 192)])
@pytest.mark.parametrize("opaque", [True, False])
def test_two_level_frames_on_both_sides_of_the_limits(bsm, ctx, oracle, w, h, opaque):
    sc = bsm.generate_instanced_scene(seed=6, instances=120, width=w, height=h, sphere_res=8, ground=16)
    if not opaque:
        sc.materials[::3, 5], sc.materials[::3, 6] = 0.5, bsm.BSM_BLEND_TRANSLUCENT
    sid = ctx.load_instanced(sc)
    det = bsm.BSM_PT_DETERMINISTIC
    imgs, st = ctx.render(sid, [sc.camera], bsm.settings(spp=1, max_segments=4, seed=8, flags=det))
    ref, ost, _ = oracle.OracleScene(sc).render(sc.camera.as_array(), spp=1, max_segments=4, seed=8, flags=det)
    assert list(st.rays_per_segment[:4]) == [int(x) for x in ost[:4]]
    assert_bits_equal(imgs[0][..., :3], ref[..., :3])
    ctx.release(sid)


@pytest.mark.parametrize("n", [1, 33, 60000, 60001])   # eight lanes per ray up to 60,000
def test_two_level_stage_entry_points_on_both_sides_of_the_limit(bsm, ctx, oracle, n):
    sc = bsm.generate_instanced_scene(seed=6, instances=120, sphere_res=8, ground=16)
    sid, osc = ctx.load_instanced(sc), oracle.OracleScene(sc)
    rays = random_rays(n, -3.0, 3.0, seed=n)
    assert np.array_equal(ctx.trace_closest(sid, rays), osc.trace(rays))
    assert np.array_equal(ctx.trace_any(sid, rays) != 0, osc.trace(rays, any_hit=True)[:, 1] != 0xFFFFFFFF)
    ctx.release(sid)
