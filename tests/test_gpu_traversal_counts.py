"""gprt_traversal_counts, the CPU walk of a batch, counts what the kernels do:
against the counters of a job whose paths end at the first surface, over as many
camera rays (other jitter: the means agree to the noise of 2^18 rays), and for
any-hit rays where every ray's work is known."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["mesh", "spheres", "cornell", "quadrics"])
def test_closest_hit_counts_are_the_kernels(ctx, name):
    import gprt
    from gprt import capi, scenes
    from test_gpu_intersect import _camera_rays
    scene = {"mesh": lambda: scenes.icosphere_scene(level=5, width=256),
             "spheres": lambda: scenes.default_style_scene(7, 256, 256),
             "cornell": lambda: scenes.cornell_baseline(256), "quadrics": lambda: scenes.quadric_scene(256)}[name]()
    scene.camera.aperture = 0.0
    scene.sampling.max_depth, scene.sampling.adaptive_min_samples = 1, 1.0
    g = gprt.GpuScene(ctx, scene)
    r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=4, seed=5,
                                                            flags=capi.JOB_COUNT_TRAVERSAL))
    r.add_samples(4)
    c = r.counters()
    rays = _camera_rays(scene, 4 * g.width * g.height, 8)
    host = np.array(g.traversal_counts(rays), dtype=np.float64) / len(rays)
    dev = np.array([c["extend_nodes"], c["extend_boxes"], c["extend_prims"]], dtype=np.float64) / c["extend_rays"]
    # a ray's counts vary by less than their mean: 5 standard errors of both means
    assert np.allclose(host, dev, rtol=5 * 2 ** 0.5 / len(rays) ** 0.5), (host, dev)
    r.close()
    g.close()


def test_any_hit_counts_the_boxes_of_a_visited_node(ctx):
    """All four children of the root are tested before the wall in its leaf is hit."""
    import gprt
    from test_gpu_intersect import _camera_rays
    from test_gpu_stack_bound import _scene
    scene = _scene()
    g = gprt.GpuScene(ctx, scene)
    rays = _camera_rays(scene, 1000, 2)
    for any_hit in (False, True):
        assert tuple(g.traversal_counts(rays, any_hit=any_hit)) == (1000, 4000, 1000)
    g.close()
