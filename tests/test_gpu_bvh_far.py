"""Device BVH builds of meshes so far from the origin that the sums of coordinates overflow: the children's centres and
their distances from the node's centre are infinite or NaN, and the lanes that share a node still agree on its slots. (Box
areas overflow too, so these meshes need the collapse that opens the largest child.) The trees' bytes are the ones recorded
for them, from the builder with a thread per 8-wide node."""
import zlib

import numpy as np
import pytest

from test_gpu_bvh_build import check_invariants, device_tree
from test_gpu_bvh_edges import soup
from test_bvh_host import decode

pytestmark = pytest.mark.gpu

# triangles -> CRC-32 of the nodes and of the leaf triangles
TREES = {
    2: (0x6dad3092, 0xecf2f3e7),
    3: (0xd46a00d2, 0x3ec2082a),
    8: (0x5e06dea8, 0x6f411efe),
    9: (0x0511ea59, 0xbb6842b7),
    33: (0x015ebb36, 0x5f5fc6c4),
    129: (0xea44e0cc, 0x78b58097),
    1000: (0x1f9ed541, 0xb12a7793),
    5000: (0x3a5576f4, 0x8b99818b),
}


@pytest.mark.parametrize("n", list(TREES))
def test_centres_that_overflow(bsm, ctx, n):
    sc = soup(bsm, "scattered", n)
    sc.positions = (2.6e38 + 0.5e38 * np.clip(sc.positions.astype(np.float64), -1.2, 1.2)).astype(np.float32)
    sid, st, nb, tb = device_tree(bsm, ctx, sc, collapse=1)
    _, tris = decode(nb, tb)
    assert np.array_equal(np.sort(tris["prim"]), np.arange(n))
    assert (zlib.crc32(nb.tobytes()), zlib.crc32(tb.tobytes())) == TREES[n]
    ctx.release(sid)


@pytest.mark.parametrize("n", [5, 33, 200, 3000])
def test_centres_that_overflow_in_part(bsm, ctx, n):
    sc = soup(bsm, "scattered", n)
    sc.positions = (1.6e38 + 0.7e38 * np.clip(sc.positions.astype(np.float64), -1.2, 1.2)).astype(np.float32)
    sid, st, nb, tb = device_tree(bsm, ctx, sc, collapse=1)
    check_invariants(sc, nb, tb, st)
    ctx.release(sid)
