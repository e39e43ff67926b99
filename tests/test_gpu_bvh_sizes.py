"""Device BVH builds at the limits of the level passes: chunks hold 1,024 references below 600,000 triangles, 2,048
below 3,000,000 and 4,096 from there on; from some 40,000 nodes in a level a block of the 8-wide passes takes more than
one tile of 32. Every tree holds each triangle once, comes out the same twice and has the bytes recorded for it (from the
builder with a thread per 8-wide node)."""
import zlib

import numpy as np
import pytest

from test_gpu_bvh_build import device_tree
from test_gpu_bvh_edges import soup
from test_bvh_host import decode

pytestmark = pytest.mark.gpu

# (kind, triangles) -> CRC-32 of the nodes and of the leaf triangles
TREES = {
    ("scattered", 1023): (0x0ffdb13c, 0x053e928f),
    ("scattered", 1024): (0xfdc8eb3d, 0x2a17d4d4),
    ("scattered", 1025): (0x1d86ffd8, 0xa4657323),
    ("scattered", 599999): (0xd27f0e18, 0xd978857e),
    ("scattered", 600000): (0xe1c04b0d, 0xb216db87),
    ("scattered", 2999999): (0xf315e87a, 0xc85aa372),
    ("scattered", 3000000): (0xb3e0a2a3, 0xeb0fff18),
    ("snapped", 600000): (0x9257ffa8, 0x020f3a26),
    ("coincident", 3000001): (0x3efad9c8, 0x43c6ed2c),
    ("duplicates", 700001): (0xf01f300d, 0x4aa2462c),
}


@pytest.mark.parametrize("kind,n", list(TREES))
def test_trees_at_the_limits_of_the_level_passes(bsm, ctx, kind, n):
    sc = soup(bsm, kind, n)
    first = None
    for _ in range(2):
        sid, st, nb, tb = device_tree(bsm, ctx, sc)
        _, tris = decode(nb, tb)
        assert np.array_equal(np.sort(tris["prim"]), np.arange(n))
        got = (zlib.crc32(nb.tobytes()), zlib.crc32(tb.tobytes()))
        assert first is None or got == first
        first = got
        ctx.release(sid)
    assert first == TREES[kind, n]
