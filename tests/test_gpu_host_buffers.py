"""Calls with host buffers around the sizes at which their staging changes
(96 KiB: 2,048 rays, 8,192 pixels of float image, 24,576 of RGBA), and
interleaved on two jobs of one context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_ray_batches_around_the_staging_limit(ctx):
    import gprt
    from gprt import scenes
    from test_gpu_intersect import _camera_rays
    scene = scenes.cornell_scene(scenes.CORNELL_SPHERES)
    g = gprt.GpuScene(ctx, scene)
    rays = _camera_rays(scene, 40000, 3)
    whole = g.intersect(rays)
    for n in (2047, 2048, 2049, 40000, 7):  # shrinking again after the large one
        assert np.array_equal(g.intersect(rays[:n]), whole[:n]), n
    g.close()


@pytest.mark.parametrize("size", [(128, 64), (129, 64), (192, 128), (193, 128)])
def test_images_around_the_staging_limit(ctx, size):
    import gprt
    from gprt import scenes
    jobs = []
    for seed in (1, 2):
        g = gprt.GpuScene(ctx, scenes.default_style_scene(seed, *size))
        jobs.append(gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=8, seed=seed)))
    for j in jobs:
        j.add_samples(3)
    for j in jobs + jobs[::-1]:
        rgb, _, _, count = j.film()
        # the device's float32 arithmetic: one reciprocal and one product per channel
        mean = (rgb * (np.float32(1.0) / count.astype(np.float32))[:, None]).reshape(j.height, j.width, 3)
        assert np.array_equal(j.image(), mean)
        want = (np.float32(255.0) * np.clip(np.sqrt(mean), 0, 1)).astype(np.uint8)
        img = j.rgba8()
        assert np.array_equal(img[..., :3], want) and (img[..., 3] == 255).all()
        assert np.array_equal(j.tile(5, 7, 21, 33), img[7:33, 5:21])
    for j in jobs:
        j.close()
        j.scene.close()
