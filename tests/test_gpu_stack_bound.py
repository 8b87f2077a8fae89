"""What fits the traversal stack, with a stack of one entry
(GPRT_BUILD_TEST_STACK_CAP): the root of this scene holds a wall and three
clusters of spheres behind it, so a ray that meets the wall needs no entry, and
one that does not needs more than one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(wall=True):
    from gprt.scene import CameraConfig, Lambertian, Quad, SamplingConfig, Scene, Sphere
    s = Scene(camera=CameraConfig(center=(0.0, 0.0, 10.0), look_at=(0.0, 0.0, 0.0), up=(0.0, 1.0, 0.0), width=64,
                                  aspect_ratio=1.0, vfov=8.0))
    s.sampling = SamplingConfig(max_depth=4, russian_roulette_min_bounces=16, adaptive_min_samples=1.0,
                                adaptive_threshold=0.0)
    s.add_uniform_infinite_light((0.5, 0.6, 0.7))
    rng = np.random.default_rng(3)
    grey = Lambertian((0.6, 0.5, 0.4))
    for z in (-10.0, -20.0, -30.0):
        for x, y, dz in rng.uniform(-3.0, 3.0, (16, 3)):
            s.add(Sphere((float(x), float(y), z + float(dz) / 3), 0.3, grey))
        for x, y in ((-4.0, -4.0), (4.0, 4.0)):  # each cluster's box holds the camera's whole view
            s.add(Sphere((x, y, z), 0.3, grey))
    if wall:
        s.add(Quad((-10.0, -10.0, 0.0), (20.0, 0.0, 0.0), (0.0, 20.0, 0.0), grey))
    return s.finalize_size()


def _both(ctx, scene, device_bvh=False):
    import gprt
    return tuple(gprt.GpuScene(ctx, scene.to_desc(), device_bvh=device_bvh, test_stack_cap=cap) for cap in (False, True))


@pytest.mark.parametrize("device_bvh", [False, True])
@pytest.mark.parametrize("any_hit", [False, True])
def test_children_behind_a_leaf_hit_take_no_room(ctx, any_hit, device_bvh):
    import gprt
    from test_gpu_intersect import _camera_rays
    scene = _scene()
    plain, capped = _both(ctx, scene, device_bvh)
    assert capped.info.n_nodes > plain.info.n_nodes  # the root's children moved apart from its leaf
    rays = _camera_rays(scene, 5000, 2)
    want = plain.intersect(rays, any_hit=any_hit)
    assert (want["prim"] != gprt.capi.NO_HIT).all()
    assert np.array_equal(capped.intersect(rays, any_hit=any_hit), want)
    plain.close()
    capped.close()
    if device_bvh:
        return  # its tree splits the spheres so that a ray without the wall needs one entry
    plain, capped = _both(ctx, _scene(wall=False))
    with pytest.raises(gprt.capi.GprtError) as e:
        capped.intersect(rays, any_hit=any_hit)
    assert e.value.code == gprt.capi.GPRT_E_BOUND
    plain.close()
    capped.close()


def test_frames_of_such_rays(ctx):
    """In every route of a path-traced frame: one launch, the wavefront, its
    simple kernels, the server."""
    import gprt
    from gprt import capi
    plain, capped = _both(ctx, _scene())

    def film(g, flags):
        r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=4, seed=2, flags=flags))
        r.add_samples(2)
        r.sync()
        f = r.film()
        r.close()
        return f

    want = film(plain, 0)
    for flags in (0, capi.JOB_COUNT_TRAVERSAL, capi.JOB_SIMPLE_EXTEND | capi.JOB_SIMPLE_SHADOW):
        for a, b in zip(film(capped, flags), want):
            assert np.array_equal(a, b), flags
    sv = gprt.RenderServer(ctx, step_paths=1 << 16)
    t = sv.submit(capped, gprt.ProgressiveConfig(initial_samples=2, max_samples_per_pixel=2, max_passes=1, seed=2))
    sv.run_until_idle()
    for a, b in zip(sv.film(t), want):
        assert np.array_equal(a, b)
    sv.close()
    plain.close()
    capped.close()


def test_a_tree_deeper_than_the_stack(ctx):
    """Spheres at distances in geometric progression: a tree of 31 levels whose
    pushes could add up to 68 entries, against the tree built on the GPU."""
    import gprt
    from gprt.scene import CameraConfig, Lambertian, Scene, Sphere
    s = Scene(camera=CameraConfig(width=32, aspect_ratio=1.0))
    rng = np.random.default_rng(0)
    grey = Lambertian((0.5, 0.5, 0.5))
    for i in range(24):
        r = 4.0 ** i
        for _ in range(200):
            d = rng.standard_normal(3)
            d *= r * (1 + 0.2 * rng.random()) / np.linalg.norm(d)
            s.add(Sphere(tuple(float(x) for x in d), 0.02 * r, grey))
    flat = s.finalize_size().to_desc()
    host, dev = gprt.GpuScene(ctx, flat), gprt.GpuScene(ctx, flat, device_bvh=True)
    n = 20000
    rays = np.zeros((n, 8), dtype=np.float32)
    rays[:, 0:3] = rng.standard_normal((n, 3)) * 4.0 ** rng.uniform(-1, 20, (n, 1))
    d = rng.standard_normal((n, 3)) - rays[:, 0:3] * 1e-3 * rng.integers(0, 2, (n, 1))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 3], rays[:, 7] = 0.001, np.inf
    for any_hit in (False, True):
        a, b = host.intersect(rays, any_hit=any_hit), dev.intersect(rays, any_hit=any_hit)
        hit = a["prim"] != gprt.capi.NO_HIT
        assert 0.2 < hit.mean() < 1.0
        assert np.array_equal(hit, b["prim"] != gprt.capi.NO_HIT)
        if not any_hit:
            assert np.array_equal(a["t"], b["t"])
    host.close()
    dev.close()
