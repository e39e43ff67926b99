"""The device refit's nodes against the host's quantiser (tlas_quantise of bvh_quant.h, compiled for the host): after
bsm_scene_update_instances every TLAS node has the bytes that the quantiser gives for its children's boxes, the instance
boxes being recomputed here in double precision, on both sides of the 256 instances up to which records and boxes are made
on the host. Transforms with negative, large and tiny coordinates and flat boxes; up
to an instance count at which a level has more than the 1,024 nodes that one block refits in rounds, and levels of their
own launches follow."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from test_bvh_host import NODE_DT

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WRAP = r"""
#include "bvh_quant.h"
extern "C" void quantise(bsm::CwNode* n, const float lo[8][3], const float hi[8][3], uint32_t used, float* nlo, float* nhi) {
    bsm::tlas_quantise(*n, lo, hi, used, nlo, nhi);
}
"""


@pytest.fixture(scope="module")
def quantise(tmp_path_factory):
    d = tmp_path_factory.mktemp("quant")
    (d / "q.cpp").write_text(WRAP)
    subprocess.run(["g++", "-std=c++20", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "bisemutum-engine_gb300", "csrc"), str(d / "q.cpp"), "-o", str(d / "q.so")], check=True)
    return C.CDLL(str(d / "q.so")).quantise


def world_boxes(lo, hi, xf):
    """The eight corners of a geometry's box in double precision, padded by 1e-5 of the magnitude and rounded outward."""
    m = xf.astype(np.float64).reshape(-1, 3, 4)
    w = []
    for c in range(8):
        p = [np.where(c >> k & 1, hi[:, k], lo[:, k]).astype(np.float64) for k in range(3)]
        w.append(np.stack([m[:, k, 0] * p[0] + m[:, k, 1] * p[1] + m[:, k, 2] * p[2] + m[:, k, 3] for k in range(3)], 1))
    mn, mx = np.min(w, 0), np.max(w, 0)
    pad = (1e-5 * np.maximum(np.abs(mn), np.abs(mx)).max(1) + 1e-30)[:, None]
    bl, bh = (mn - pad).astype(np.float32), (mx + pad).astype(np.float32)
    for _ in range(3):
        bl = np.where(bl.astype(np.float64) > mn - pad, np.nextafter(bl, np.float32(-np.inf)), bl)
        bh = np.where(bh.astype(np.float64) < mx + pad, np.nextafter(bh, np.float32(np.inf)), bh)
    return bl, bh


def moved_transforms(rng, n, spread):
    q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    scale = 10.0 ** rng.uniform(-3, 1, (n, 1, 3))
    t = rng.uniform(-1, 1, (n, 3, 1)) * spread
    t[::7] *= 1e-4
    xf = np.concatenate([q * scale, t], 2).astype(np.float32)
    xf[::5, :, :3] = np.eye(3, dtype=np.float32) * xf[::5, 0, :1, None]   # along the axes: flat geometry stays flat
    xf[::5, :, :3] += np.where(np.eye(3) == 1, np.float32(0.01), np.float32(0.0))
    return xf.reshape(n, 12)


@pytest.mark.parametrize("n,spread", [(1, 3.0), (256, 5.0), (257, 5.0), (300, 0.5), (300, 2e4), (20000, 30.0)])
def test_refitted_nodes_have_the_quantisers_bytes(bsm, ctx, quantise, n, spread):
    rng = np.random.default_rng(n + int(spread))
    box = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32)
    geoms = [bsm.GeometryData(box * np.float32(0.3), np.array([[0, 1, 3], [4, 6, 7], [0, 4, 5]], np.uint32), None),
             bsm.GeometryData(box[[0, 2, 6]] * np.float32([1, 0, 2]), np.array([[0, 1, 2]], np.uint32), None),  # flat
             bsm.GeometryData(box[[1, 3, 5]] + np.float32(7.5), np.array([[0, 1, 2]], np.uint32), None)]
    kind = rng.integers(0, 3, n)
    first = np.tile(np.eye(3, 4, dtype=np.float32), (n, 1, 1))   # instances of one size: their tree is of even depth
    first[:, :, 3] = rng.uniform(-30, 30, (n, 3))
    sc = bsm.InstancedSceneData(geoms, kind.astype(np.uint32), np.zeros(n, np.uint32), first.reshape(n, 12),
                                np.array([[0.5, 0.5, 0.5, 0.5, 0.0]], np.float32),
                                np.array([[0.0, 1.0, 0.0, 1.0, 1.0, 1.0]], np.float32), bsm.BSM_SKY_CONSTANT,
                                (0.3, 0.3, 0.3), None, bsm.make_camera((0, 0, 9), (0, 0, -1), width=16, height=16))
    sid = ctx.load_instanced(sc)
    st = ctx.build_bvh(sid)
    before = ctx.download_bvh(sid, st)[0].copy()
    xf = moved_transforms(rng, n, spread)
    ctx.update_instances(sid, xf)
    nb, ib = ctx.download_bvh(sid, st)
    ctx.release(sid)

    insts = ib.view(np.uint32).reshape(n, 32)
    order = insts[:, 30]   # leaf -> instance
    assert np.array_equal(np.sort(order), np.arange(n))
    assert np.array_equal(insts[:, 12:24], xf.view(np.uint32)[order])
    glo, ghi = (np.array([f(g.positions, 0) for g in geoms], np.float32)[kind] for f in (np.min, np.max))
    bl, bh = world_boxes(glo, ghi, xf)
    bl, bh = bl[order], bh[order]

    nodes = before.view(NODE_DT)
    level = np.zeros(len(nodes), int)
    lo, hi = np.zeros((len(nodes), 3), np.float32), np.zeros((len(nodes), 3), np.float32)
    raw = before.reshape(-1, 80).copy()
    f32p = C.POINTER(C.c_float)
    for ni in range(len(nodes) - 1, -1, -1):   # children come after their parents
        im, tm = int(nodes[ni]["imask"]), int(nodes[ni]["tri_mask"])
        cl, ch = np.zeros((8, 3), np.float32), np.zeros((8, 3), np.float32)
        used, child, leaf = 0, int(nodes[ni]["child_base"]), int(nodes[ni]["tri_base"])
        for s in range(8):
            if im >> s & 1:
                cl[s], ch[s] = lo[child], hi[child]
                child += 1
            elif tm >> 2 * s & 3:
                cl[s], ch[s] = bl[leaf], bh[leaf]
                leaf += 1
            else:
                continue
            used |= 1 << s
        quantise(raw[ni].ctypes.data_as(C.c_void_p), cl.ctypes.data_as(C.c_void_p), ch.ctypes.data_as(C.c_void_p),
                 C.c_uint32(used), lo[ni].ctypes.data_as(f32p), hi[ni].ctypes.data_as(f32p))
    for ni in range(len(nodes)):
        c = int(nodes[ni]["child_base"])
        level[c:c + bin(int(nodes[ni]["imask"])).count("1")] = level[ni] + 1
    if n == 20000:
        assert np.bincount(level).max() > 1024   # a level that several blocks refit
    got = nb.reshape(-1, 80)
    bad = np.argwhere(got != raw)
    assert bad.size == 0, f"{len(bad)} bytes of {len(np.unique(bad[:, 0]))} nodes differ, first {bad[0]}"
