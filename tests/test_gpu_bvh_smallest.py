"""The smallest device builds queue no more levels than such meshes can have."""
import pytest

from test_gpu_bvh_edges import soup

pytestmark = pytest.mark.gpu


def build_ms(ctx, sid, times=20):
    return min(ctx.build_bvh(sid).build_ms for _ in range(times))


def test_two_triangles_build_without_empty_levels(bsm, ctx):
    """Two triangles make one node: the two launches of its level, not those of twelve levels, which take as long as the
    rest of the build of a two-level tree of 33."""
    a, b = ctx.upload(soup(bsm, "scattered", 2)), ctx.upload(soup(bsm, "scattered", 33))
    try:
        assert build_ms(ctx, a) < 0.7 * build_ms(ctx, b)
    finally:
        ctx.release(a)
        ctx.release(b)


@pytest.mark.parametrize("kind", ["scattered", "coincident"])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33])   # one level, four and twelve are queued first
@pytest.mark.parametrize("collapse,max_leaf", [(0, 0), (0, 1), (1, 1), (1, 2)])
def test_batches_of_levels_reach_every_triangle(bsm, ctx, kind, n, collapse, max_leaf):
    from test_gpu_bvh_build import check_invariants, device_tree
    sc = soup(bsm, kind, n)
    sid, st, nb, tb = device_tree(bsm, ctx, sc, collapse=collapse, max_leaf=max_leaf)
    check_invariants(sc, nb, tb, st)
    ctx.release(sid)
