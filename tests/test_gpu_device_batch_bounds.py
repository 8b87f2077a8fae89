"""Device ray batches report an overflowed stack in the hit records alone."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_overflowed_rays_are_marked(ctx):
    torch = pytest.importorskip("torch")
    import gprt
    from gprt import capi, scenes
    scene = scenes.icosphere_scene(level=4, width=40)
    rays = scenes.ray_batch(*scenes.icosphere(4), 4096, seed=3)
    plain = gprt.GpuScene(ctx, scene.to_desc())
    want = plain.intersect(rays)
    plain.close()
    g = gprt.GpuScene(ctx, scene.to_desc(), test_stack_cap=True)
    d, st = torch.from_numpy(rays).cuda(), torch.cuda.Stream()
    h = torch.zeros((len(rays), 4), device="cuda")
    torch.cuda.synchronize()
    ctx.check(ctx.lib.gprt_intersect(g.h, C.c_void_p(d.data_ptr()), len(rays), capi.CLOSEST, C.c_void_p(h.data_ptr()),
                                     C.c_void_p(st.cuda_stream)))
    st.synchronize()
    got = h.cpu().numpy()
    prim = got.view(np.uint32)[:, 1]
    over = prim == capi.BOUND_HIT
    assert over.any() and (got[over, 0] == -1).all()
    assert np.array_equal(prim[~over], want["prim"][~over])
    g.close()
