"""Device BVH builds at the sizes where the builder's kernels change: 32 triangles (one lane each) and 128 (one
warp) for the small nodes, 4,096 per chunk of a level, with scattered, snapped and coincident centroids.  Every tree
keeps the invariants and traverses to the oracle's hits, and its bytes are the ones recorded for it: the kernels
may change, the tree is defined by the binned SAH splits and the collapse."""
import zlib

import numpy as np
import pytest

from conftest import random_rays
from test_gpu_bvh_build import check_invariants, device_tree

pytestmark = pytest.mark.gpu

# (kind, triangles, collapse, max_leaf) -> CRC-32 of the nodes and of the leaf triangles
TREES = {
    ("scattered", 5, 0, 0): (0x8adb6459, 0x14753299),
    ("scattered", 31, 0, 0): (0x6c49aaed, 0xc640ac9f),
    ("scattered", 32, 1, 2): (0x0d3b8a5c, 0xefb02bf8),
    ("scattered", 33, 0, 0): (0xd45dbdf8, 0x36da1ead),
    ("scattered", 65, 1, 1): (0xb1ce7d32, 0x8cd4a068),
    ("scattered", 127, 0, 1): (0xbd950dd5, 0xc716d2f2),
    ("scattered", 129, 0, 0): (0x2a2cc819, 0x2dd549ac),
    ("scattered", 4097, 0, 0): (0x22067938, 0xae1efd10),
    ("scattered", 8192, 1, 2): (0x5c4a6947, 0xd6c75782),
    ("scattered", 20011, 0, 0): (0xa92e2560, 0xa247bcb5),
    ("snapped", 5, 0, 0): (0xbebda157, 0x0c106cc7),
    ("snapped", 31, 0, 0): (0x95994f0f, 0xfae34283),
    ("snapped", 32, 1, 2): (0xe15178b3, 0x1c79eb15),
    ("snapped", 33, 0, 0): (0xa62ba7b9, 0xf04470ab),
    ("snapped", 65, 1, 1): (0x498d0145, 0xa74a8843),
    ("snapped", 127, 0, 1): (0x6f735c61, 0x85e0ff00),
    ("snapped", 129, 0, 0): (0x309bade6, 0x669f9b5b),
    ("snapped", 4097, 0, 0): (0x9af41cec, 0xbf789f9b),
    ("snapped", 8192, 1, 2): (0xfa57dce2, 0xbba81563),
    ("snapped", 20011, 0, 0): (0x9f946d8b, 0xf9b237cc),
    ("coincident", 5, 0, 0): (0xf3105dd8, 0xced80d77),
    ("coincident", 31, 0, 0): (0xe375873a, 0xef515036),
    ("coincident", 32, 1, 2): (0x2a2de787, 0x7ecff2c3),
    ("coincident", 33, 0, 0): (0xd8887feb, 0xdcc1d59b),
    ("coincident", 65, 1, 1): (0xde36dbfd, 0x74eb4b05),
    ("coincident", 127, 0, 1): (0xa6f59d79, 0x00407f93),
    ("coincident", 129, 0, 0): (0xba17e8e9, 0xfdcd6ad1),
    ("coincident", 4097, 0, 0): (0xb53b56ec, 0x9c6098fd),
    ("coincident", 8192, 1, 2): (0x3bca4fef, 0x1da1461a),
    ("coincident", 20011, 0, 0): (0x437e1c52, 0x02b4b855),
    ("duplicates", 5, 0, 0): (0xa31eaeba, 0x62141b93),
    ("duplicates", 31, 0, 0): (0xaec13928, 0x36e4ac19),
    ("duplicates", 32, 1, 2): (0xdefb8e20, 0xba087b1e),
    ("duplicates", 33, 0, 0): (0x84b1bbcd, 0xaef4518c),
    ("duplicates", 65, 1, 1): (0xecf339a9, 0x7c085ba1),
    ("duplicates", 127, 0, 1): (0xbd7f3240, 0x324a88dc),
    ("duplicates", 129, 0, 0): (0xe3cc5402, 0xc708cc27),
    ("duplicates", 4097, 0, 0): (0x0c3c0d46, 0x6c5c0a17),
    ("duplicates", 8192, 1, 2): (0x0a1f7e82, 0x5758b9dc),
    ("duplicates", 20011, 0, 0): (0x0e542249, 0x4de61c0d),
}


def soup(bsm, kind, n):
    g = np.random.default_rng(1000 + n)
    c = g.uniform(-1, 1, (n, 1, 3))
    if kind == "coincident":
        c[:] = 0.25
    if kind == "duplicates":
        c = c[g.integers(0, max(1, n // 4), n)]
    p = c + g.normal(0, 0.02, (n, 3, 3))
    if kind == "snapped":
        p = np.round(p * 16) / 16
    return bsm.SceneData(p.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3),
                         np.zeros(n, np.uint32), np.array([[0.5, 0.5, 0.5, 0.5, 0.0]], np.float32),
                         np.array([[0.0, 1.0, 0.0, 1.0, 1.0, 1.0]], np.float32), bsm.BSM_SKY_CONSTANT, (0.3, 0.3, 0.3))


@pytest.mark.parametrize("kind,n,collapse,max_leaf", list(TREES))
def test_trees_at_the_builders_limits(bsm, ctx, oracle, kind, n, collapse, max_leaf):
    sc = soup(bsm, kind, n)
    sid, st, nb, tb = device_tree(bsm, ctx, sc, collapse=collapse, max_leaf=max_leaf)
    check_invariants(sc, nb, tb, st)
    rays = random_rays(2000, -1.0, 1.0, seed=n)
    assert np.array_equal(ctx.trace_closest(sid, rays)[:, :2], oracle.OracleScene(sc).trace(rays)[:, :2])
    assert (zlib.crc32(nb.tobytes()), zlib.crc32(tb.tobytes())) == TREES[kind, n, collapse, max_leaf]
    ctx.release(sid)
