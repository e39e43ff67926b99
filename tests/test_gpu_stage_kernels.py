"""The stage entry points on both sides of every limit between their kernels (eight lanes per ray, a ray per thread, lanes
that take new rays), in one level and in two, with few, some and many instances: incoherent rays, a camera's, and the two
in turns, so that a warp finds its next 32 rays alike or not. Every hit equals the oracle's."""
import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu

LANES = 152 * 8 * 128   # rays that 152 SMs hold with a ray per thread


def mixed_rays(n, lo, hi, seed):
    """Thirds: incoherent; a camera's, row by row; stretches of 1 to 100 rays of either kind."""
    r = random_rays(n, lo, hi, seed=seed)
    w = max(1, int((n / 3) ** 0.5))
    y, x = np.divmod(np.arange(n), w)
    d = np.stack([(2 * (x + 0.5) / w - 1) * 0.6, -0.3 - (2 * ((y % w) + 0.5) / w - 1) * 0.6, -np.ones(n)], 1)
    cam = r.copy()
    cam[:, 0:3] = [(lo + hi) / 2, lo + (hi - lo) * 0.9, hi]
    cam[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    g = np.random.default_rng(seed)
    runs = np.repeat(g.integers(0, 2, n), g.integers(1, 100, n))[:n].astype(bool)
    pick = np.where(np.arange(n) < n // 3, False, np.where(np.arange(n) < 2 * n // 3, True, runs))
    r[pick] = cam[pick]
    r[n // 2, 4:7] = 0.0        # one that is not traced, among rays that are alike
    return r


CASES = [("room", n) for n in (40000, 40001, LANES, LANES + 1, LANES + 31)] + [("veil", n) for n in (40001, 2 * LANES, 2 * LANES + 1)]
CASES += [(8, n) for n in (25000, 25001, 32000, 32001, 100000, 100001, 400000, 400001)]
CASES += [(64, n) for n in (40000, 40001, 100000, 100001)] + [(500, n) for n in (60000, 60001)]


@pytest.mark.parametrize("scene,n", CASES)
def test_both_sides_of_every_limit(bsm, ctx, oracle, scene, n):
    if isinstance(scene, int):
        sc = bsm.generate_instanced_scene(seed=6, instances=scene - 1, sphere_res=8, ground=16)   # and the ground
        assert len(sc.inst_geometry) == scene
        sid, lo, hi = ctx.load_instanced(sc), -3.0, 3.0
    else:
        sc = bsm.generate_scene(bsm.BSM_SCENE_ROOM, seed=12)
        if scene == "veil":
            sc.materials[::2, 5], sc.materials[::2, 6] = 0.5, bsm.BSM_BLEND_TRANSLUCENT
        sid, lo, hi = ctx.load_scene(sc), 0.0, 1.0
    osc, rays = oracle.OracleScene(sc), mixed_rays(n, lo, hi, seed=n)
    for _ in range(2):   # the second call starts from the counter that the first one left
        assert np.array_equal(ctx.trace_closest(sid, rays), osc.trace(rays))
        assert np.array_equal(ctx.trace_any(sid, rays) != 0, osc.trace(rays, any_hit=True)[:, 1] != 0xFFFFFFFF)
    ctx.release(sid)
