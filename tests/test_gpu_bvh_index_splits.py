"""Splits by index, of triangles whose centroids are one point: their boxes are merged once per chunk of references, so
such a mesh builds about as fast as a scattered one of its size (before: six global atomics per reference and level, four
times as long). The trees' bytes are the ones recorded for them."""
import zlib

import numpy as np
import pytest

from test_gpu_bvh_build import device_tree
from test_gpu_bvh_edges import soup
from test_bvh_host import decode

pytestmark = pytest.mark.gpu

# triangles -> CRC-32 of the nodes and of the leaf triangles
TREES = {
    129: (0x87fa0b24, 0x38e42941),
    5000: (0x34356de7, 0x9ebdb009),
    20000: (0xbc308c59, 0x18c43e68),
    250000: (0x76881fc6, 0x75230913),
    600001: (0x2fc73584, 0xa1823215),
}


def star(bsm, n):
    """Triangles through one point: every box is centred on it exactly (offsets in steps of 2^-13)."""
    sc = soup(bsm, "scattered", n)
    g = np.random.default_rng(1000 + n)
    g.uniform(-1, 1, (n, 1, 3)), g.normal(0, 0.02, (n, 3, 3))   # the scattered mesh's draws come first
    d = g.integers(1, 1024, (n, 3)) / 8192.0
    sc.positions = np.stack([0.25 + d, 0.25 - d, 0.25 + 0 * d], 1).reshape(-1, 3).astype(np.float32)
    return sc


@pytest.mark.parametrize("n", list(TREES))
def test_trees_of_splits_by_index(bsm, ctx, n):
    sid, st, nb, tb = device_tree(bsm, ctx, star(bsm, n))
    _, tris = decode(nb, tb)
    assert np.array_equal(np.sort(tris["prim"]), np.arange(n))
    assert (zlib.crc32(nb.tobytes()), zlib.crc32(tb.tobytes())) == TREES[n]
    ctx.release(sid)


def build_ms(ctx, sid, times=5):
    return min(ctx.build_bvh(sid).build_ms for _ in range(times))


def test_splits_by_index_take_no_longer_than_binned_ones(bsm, ctx):
    n = 600001
    a, b = ctx.upload(star(bsm, n)), ctx.upload(soup(bsm, "scattered", n))
    try:
        assert build_ms(ctx, a) < 1.5 * build_ms(ctx, b)   # one pass over the references a level, as the binned one
    finally:
        ctx.release(a)
        ctx.release(b)
