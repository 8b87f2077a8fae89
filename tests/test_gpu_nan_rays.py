"""Rays that are not numbers: the primitives of a leaf accept them at a distance
that is not a number either, with which no box can be compared.  Such a ray ends
after the nodes on its stack, with the hit that it had before the traversal
deferred its leaves, and takes no longer than another."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# level of the icosphere, columns that are not numbers, any hit -> hits at a
# distance that is not a number, and the sum of the primitive ids
EXPECTED = {
    (4, "dx", False): (1940, 9259957041183), (4, "dx", True): (1940, 9259957038219),
    (4, "ox", False): (4091, 21487084651), (4, "ox", True): (4091, 21487063772),
    (4, "o", False): (4096, 20971520), (4, "o", True): (4096, 20971520),
    (5, "dx", False): (1892, 9466138193443), (5, "dx", True): (1892, 9466138191159),
    (5, "ox", False): (4089, 30119633692), (5, "ox", True): (4089, 30119613211),
    (5, "o", False): (4096, 83886080), (5, "o", True): (4096, 83886080),
}
COLUMNS = {"d": [4, 5, 6], "dx": [4], "o": [0, 1, 2], "ox": [0]}


def _rays(level, n, kind):
    from gprt import scenes
    rays = scenes.ray_batch(*scenes.icosphere(level), n, seed=3)
    for c in COLUMNS[kind]:
        rays[:, c] = np.nan
    return rays


@pytest.mark.parametrize("level", [4, 5])
def test_hits_of_rays_that_are_not_numbers(ctx, level):
    import gprt
    from gprt import scenes
    g = gprt.GpuScene(ctx, scenes.icosphere_scene(level=level, width=64))
    for kind in ("dx", "ox", "o"):
        rays = _rays(level, 4096, kind)
        for any_hit in (False, True):
            h = g.intersect(rays, any_hit=any_hit)
            got = int(np.isnan(h["t"]).sum()), int(h["prim"].astype(np.int64).sum())
            assert got == EXPECTED[level, kind, any_hit], (kind, any_hit)
    g.close()


def test_they_cost_no_more_than_others(ctx):
    import gprt
    from gprt import scenes
    level, n = 6, 65536
    g = gprt.GpuScene(ctx, scenes.icosphere_scene(level=level, width=64))

    def took(rays):
        best = np.inf
        for _ in range(4):
            t = time.perf_counter()
            g.intersect(rays)
            best = min(best, time.perf_counter() - t)
        return best

    usual = took(scenes.ray_batch(*scenes.icosphere(level), n, seed=3))
    for kind in COLUMNS:
        # the whole tree, which has 20,000 nodes, takes hundreds of times as long
        assert took(_rays(level, n, kind)) < 4 * usual + 2e-3, kind
    g.close()
