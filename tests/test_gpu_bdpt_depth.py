"""BDPT at depth 0: no ray is traced, so the film is black with its samples
counted, as the oracle's; on working memory that an earlier job has written."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _film(ctx, scene, depth, spp, chunk):
    import gprt
    scene.sampling.max_depth = depth
    scene.sampling.adaptive_min_samples = 1.0
    g = gprt.GpuScene(ctx, scene)
    r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=8, seed=3, chunk_paths=chunk),
                                  gprt.BDPTIntegrator())
    r.add_samples(spp)
    r.sync()
    f = r.film()
    r.close()
    g.close()
    return f


@pytest.mark.parametrize("chunk", [0, 997])
@pytest.mark.parametrize("name", ["boxes", "spheres", "spot"])
def test_depth_zero_is_black(ctx, oracle, name, chunk):
    from gprt import scenes
    make = {"boxes": lambda: scenes.cornell_boxes_bdpt(40), "spheres": lambda: scenes.default_style_scene(5, 41, 30),
            "spot": lambda: scenes.spot_scene(40)}[name]
    _film(ctx, make(), 6, 3, chunk)
    rgb, lum, lum2, count = _film(ctx, make(), 0, 3, chunk)
    assert not rgb.any() and not lum.any() and not lum2.any()
    assert (count == 3).all()
    flat = make()
    flat.sampling.max_depth = 0
    o = oracle.OracleRenderer(oracle.OracleScene(flat.to_desc()), 1, max_spp=3, max_passes=1, seed=3)
    o.render_pass(1)
    assert not o.film()[0].any()
