"""Small BDPT chunks (subpaths in one launch, strategies in one) against the
wavefront that larger chunks take: the luminance sums, which hold everything
but the light-tracing splats (float atomics), around one sample per warp, one
per lane and the largest small chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152
WARPS = SMS * 16
SMALL = SMS * 1024


def _scene(name, depth):
    from gprt import scenes
    from gprt.scene import CameraConfig
    s = {"boxes": lambda: scenes.cornell_boxes_bdpt(400),
         "spot": lambda: scenes.spot_scene(340),
         "spheres": lambda: scenes.default_style_scene(5, 401, 390),
         "textures": lambda: scenes.texture_test_scene(CameraConfig(width=540)),
         "mesh": lambda: scenes.icosphere_scene(level=3, width=400)}[name]()
    s.sampling.max_depth = depth
    s.sampling.adaptive_min_samples = 1.0
    return s


@pytest.mark.parametrize("name,depth", [("boxes", 6), ("spot", 6), ("spheres", 6), ("textures", 6), ("mesh", 6),
                                        ("boxes", 1), ("spheres", 1), ("boxes", 17), ("spheres", 12)])
def test_small_chunks_equal_the_wavefronts(ctx, name, depth):
    import gprt
    g = gprt.GpuScene(ctx, _scene(name, depth))
    assert g.width * g.height > SMALL  # one chunk of all pixels takes the wavefront

    def film(chunk):
        r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=4, seed=3, chunk_paths=chunk),
                                      gprt.BDPTIntegrator())
        r.add_samples(1)
        f = r.film()
        r.close()
        return f

    _, lum, lum2, count = film(0)
    for chunk in (997, WARPS - 1, 32 * WARPS + 1, SMALL, SMALL + 1):
        _, l, l2, c = film(chunk)
        assert np.array_equal(c, count)
        assert np.array_equal(l, lum), chunk
        assert np.array_equal(l2, lum2), chunk
    g.close()
