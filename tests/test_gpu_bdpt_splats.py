"""The light-tracing part of a BDPT film (splats, added by float atomics): small
chunks, whose strategies share one launch, against the wavefront's, to what the
order of the additions leaves.  The luminance sums hold everything but it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,depth", [("boxes", 6), ("spot", 6), ("spheres", 5), ("boxes", 12)])
def test_small_chunks_splat_as_the_wavefront(ctx, name, depth):
    import torch
    import gprt
    from gprt import scenes
    small = torch.cuda.get_device_properties(0).multi_processor_count * 1024
    width = int((small / (0.69 if name == "spot" else 1.0)) ** 0.5) + 24
    s = {"boxes": lambda: scenes.cornell_boxes_bdpt(width), "spot": lambda: scenes.spot_scene(width),
         "spheres": lambda: scenes.default_style_scene(5, width, width)}[name]()
    s.sampling.max_depth, s.sampling.adaptive_min_samples = depth, 1.0
    g = gprt.GpuScene(ctx, s)
    assert g.width * g.height > small

    def film(chunk):
        r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=4, seed=3, chunk_paths=chunk),
                                      gprt.BDPTIntegrator())
        r.add_samples(2)
        f = r.film()
        r.close()
        return f

    rgb, lum, _, _ = film(0)  # one chunk a sample: the wavefront
    splat = rgb @ np.array([0.2126, 0.7152, 0.0722]) - lum
    assert splat.max() > 1e-3  # there is light tracing to compare
    for chunk in (small, 20011):
        got = film(chunk)
        assert np.array_equal(got[1], lum)
        # a pixel's splats are at most a few hundred float32 additions in another order
        assert np.allclose(got[0], rgb, rtol=1e-4, atol=1e-4 * splat.max())
    g.close()
