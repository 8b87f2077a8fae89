"""Small wavefronts rendered path by path in one launch give the films of the
bounce-by-bounce wavefront (which a job that counts its traversal runs), bit
for bit: around one path per warp, one per lane and the largest such chunk, and
over the materials, lights, textures and Russian roulette."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152
WARPS = SMS * 16


def _film(g, spp, flags=0, chunk=0):
    import gprt
    r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=64, seed=9, flags=flags,
                                                            chunk_paths=chunk))
    for s in spp:  # the later samples start from a film that holds some
        r.add_samples(s)
    f = r.film()
    r.close()
    return f


def _same(ctx, scene, spp, chunks):
    import gprt
    from gprt import capi
    g = gprt.GpuScene(ctx, scene)
    want = _film(g, spp, flags=capi.JOB_COUNT_TRAVERSAL)
    for chunk in chunks:
        for a, b in zip(_film(g, spp, chunk=chunk), want):
            assert np.array_equal(a, b), chunk
    g.close()


def _scene(name):
    from gprt import scenes
    from gprt.scene import CameraConfig
    s = {"cornell": lambda: scenes.cornell_baseline(96),
         "textures": lambda: scenes.texture_test_scene(CameraConfig(width=97)),
         "textured_mesh": lambda: scenes.textured_mesh_scene(96),
         "spheres": lambda: scenes.default_style_scene(5, 101, 83),
         "layered": lambda: scenes.default_scene(CameraConfig(width=96)),
         "mix": lambda: scenes.sphere_grid_scene(8, "mixed", CameraConfig(width=96)),
         "point_spot": lambda: scenes.spot_scene(90, True),
         "disc_light": lambda: scenes.quadric_scene(90, 8, True)}[name]()
    s.sampling.adaptive_min_samples = 1.0
    return s


@pytest.mark.parametrize("roulette", [False, True])
@pytest.mark.parametrize("name", ["cornell", "textures", "textured_mesh", "spheres", "layered", "mix", "point_spot",
                                  "disc_light"])
def test_films_equal_the_wavefronts(ctx, name, roulette):
    scene = _scene(name)
    scene.sampling.max_depth, scene.sampling.russian_roulette_min_bounces = (20, 2) if roulette else (6, 16)
    _same(ctx, scene, (3, 2), [0, 33, WARPS - 1, WARPS + 1])


@pytest.mark.parametrize("name", ["cornell", "spheres"])
def test_chunk_edges(ctx, name):
    from gprt import scenes
    scene = scenes.cornell_baseline(490) if name == "cornell" else scenes.default_style_scene(5, 800, 790)
    most = SMS * (1536 if name == "cornell" else 4096)
    _same(ctx, scene, (1,), [SMS * 256, SMS * 256 + 1, 32 * WARPS - 1, 32 * WARPS + 1, most, most + 1])


@pytest.mark.parametrize("depth", [0, 1])
def test_shallow_paths(ctx, depth):
    scene = _scene("cornell")
    scene.sampling.max_depth = depth
    _same(ctx, scene, (2,), [0])


def test_adaptive_pixel_lists(ctx):
    """A pass whose rounds take one sample of the pixels still active."""
    import gprt
    from gprt import capi
    scene = _scene("layered")
    scene.sampling.adaptive_min_samples, scene.sampling.adaptive_threshold = 0.15, 0.05
    g = gprt.GpuScene(ctx, scene)
    got = []
    for flags in (0, capi.JOB_COUNT_TRAVERSAL):
        r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=16, max_passes=3, seed=4, flags=flags))
        for p in (1, 2, 3):
            r.render_pass(p)
        got.append(r.film())
        r.close()
    assert got[0][3].min() < got[0][3].max()  # some pixels stopped earlier
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    g.close()
