"""The traversal's dealing of rays to warps and its two forms (one-node scenes
and trees): a ray's hit does not depend on the batch it comes in, and agrees
with the oracle by the rule of test_gpu_intersect."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rays per warp of a full grid: fewer than one, one, a part of a chunk, a
# whole chunk (64) and the first ray of the second
WARPS = 152 * 8 * 4
SIZES = [1, 31, 33, WARPS - 1, WARPS + 1, 20 * WARPS + 7, 64 * WARPS - 1, 64 * WARPS + 1]


def _scene(name):
    from gprt import scenes
    if name == "one_node_quads":
        return scenes.cornell_baseline(64)
    if name == "one_node_mixed":
        return scenes.texture_test_scene()
    if name == "spheres":
        return scenes.default_style_scene(7, 64, 64)
    return scenes.icosphere_scene(level=4, width=64)


@pytest.mark.parametrize("name", ["one_node_quads", "one_node_mixed", "spheres", "mesh"])
@pytest.mark.parametrize("any_hit", [False, True])
def test_hits_do_not_depend_on_the_batch(ctx, oracle, name, any_hit):
    import gprt
    from test_gpu_intersect import _camera_rays, _compare
    scene = _scene(name)
    rays = _camera_rays(scene, SIZES[-1], 5)
    g = gprt.GpuScene(ctx, scene)
    whole = g.intersect(rays, any_hit=any_hit)
    for n in SIZES[:-1]:
        assert np.array_equal(g.intersect(rays[:n], any_hit=any_hit), whole[:n]), n
    g.close()
    # the oracle's rule: at most max(2, 1e-4 n) rays graze a silhouette otherwise
    if any_hit:
        g_hit, o_hit = _compare(ctx, oracle, scene, rays[:4000], any_hit=True)
        assert (g_hit != o_hit).sum() <= 2
    else:
        r = _compare(ctx, oracle, scene, rays[:4000])
        assert max(r["hit_disagree"], r["bad_prim"], r["rel_bad"]) <= 2, r
