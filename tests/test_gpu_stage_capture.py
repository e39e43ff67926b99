"""Stage entry points captured into a caller's graph: a replay shares nothing with the calls around it, nor with a replay
of the same captured call from a second graph. Replays run beside direct calls of the same context and beside one another,
after more direct calls than any ring of counters would hold; every ray gets the oracle's hit."""
import ctypes as C

import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MISS = 0xFFFFFFFF
CAMERA = (200, 120)   # 24,000 pixels: primary outputs with eight lanes per ray


@pytest.fixture(scope="module")
def own(bsm):
    c = bsm.Context(0)
    yield c
    c.set_stream(None)
    c.close()


def capture(ctx, stream, call):
    g = torch.cuda.CUDAGraph()
    ctx.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=stream):
        call()
    ctx.set_stream(None)
    return g


# on both sides of the limits between eight lanes and one lane per ray, and of the rays that fit the GPU at once
@pytest.mark.parametrize("two_level,n", [(False, 9000), (False, 39999), (False, 120001), (False, 300007),
                                         (False, 1300003), (True, 9000), (True, 59999), (True, 300007)])
def test_replays_share_no_counter_with_other_calls(bsm, own, oracle, two_level, n):
    ctx, L = own, bsm.lib()
    if two_level:
        sc = bsm.generate_instanced_scene(seed=6, instances=120, sphere_res=8, ground=16)
        sid, osc, rays = ctx.load_instanced(sc), oracle.OracleScene(sc), random_rays(n, -3.0, 3.0, seed=n)
    else:
        sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=12)
        sid, osc, rays = ctx.load_scene(sc), oracle.OracleScene(sc), random_rays(n, 0.0, 1.0, seed=n)
    ref, anyref = osc.trace(rays), osc.trace(rays, any_hit=True)[:, 1] != MISS
    dev = torch.from_numpy(rays).cuda()
    hits = [torch.empty((n, 4), dtype=torch.int32, device="cuda") for _ in range(3)]
    occ = torch.empty(n, dtype=torch.uint8, device="cuda")
    few = torch.from_numpy(rays[:64]).cuda()
    few_hits = torch.empty((64, 4), dtype=torch.int32, device="cuda")

    def closest(k):
        ctx.check(L.bsm_trace_closest(ctx.h, sid, dev.data_ptr(), n, hits[k].data_ptr(), bsm.BSM_DEVICE))

    def occluded():
        ctx.check(L.bsm_trace_any(ctx.h, sid, dev.data_ptr(), n, occ.data_ptr(), bsm.BSM_DEVICE))

    streams = [torch.cuda.Stream() for _ in range(3)]
    graphs = [capture(ctx, streams[0], lambda: closest(0)), capture(ctx, streams[1], occluded)]
    for _ in range(1030):
        ctx.check(L.bsm_trace_closest(ctx.h, sid, few.data_ptr(), 64, few_hits.data_ptr(), bsm.BSM_DEVICE))
    ctx.sync()
    for _ in range(3):
        for h in hits:
            h.fill_(-2)
        occ.fill_(7)
        torch.cuda.synchronize()
        ctx.set_stream(streams[2].cuda_stream)
        for g, st in zip(graphs, streams):
            with torch.cuda.stream(st):
                g.replay()
        closest(1)
        closest(2)
        ctx.sync()
        torch.cuda.synchronize()
        for h in hits:
            assert np.array_equal(h.cpu().numpy().view(np.uint32), ref)
        assert np.array_equal(occ.cpu().numpy() != 0, anyref) and int(occ.max()) <= 1
    ctx.set_stream(None)
    assert np.array_equal(ctx.trace_closest(sid, rays), ref)   # and later direct calls start from a clean counter
    del graphs
    ctx.release(sid)


def test_captured_primary_outputs(bsm, own, oracle):
    ctx, L = own, bsm.lib()
    w, h = CAMERA
    sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=13, width=w, height=h)
    sid, cam = ctx.load_scene(sc), sc.camera
    _, _, ref = oracle.OracleScene(sc).primary(cam.as_array())
    pos = [torch.empty((h, w, 4), dtype=torch.float32, device="cuda") for _ in range(2)]

    def primary(k):
        out = bsm.PrimaryOutput()
        out.hit_positions = pos[k].data_ptr()
        out.location = bsm.BSM_DEVICE
        ctx.check(L.bsm_render_primary(ctx.h, sid, C.byref(cam), None, 0.0, 0.0, C.byref(out)))

    st, other = torch.cuda.Stream(), torch.cuda.Stream()
    g = capture(ctx, st, lambda: primary(0))
    for p in pos:
        p.fill_(-2.0)
    torch.cuda.synchronize()
    ctx.set_stream(other.cuda_stream)
    with torch.cuda.stream(st):
        g.replay()
    primary(1)
    ctx.sync()
    torch.cuda.synchronize()
    ctx.set_stream(None)
    for p in pos:
        assert np.array_equal(p.cpu().numpy().view(np.uint32).reshape(-1), ref.view(np.uint32).reshape(-1))
    del g
    ctx.release(sid)
