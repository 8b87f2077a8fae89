"""The device bounds of the wavefronts: frames of a few thousand paths take one
launch, so these ask for the wavefront (a job that counts its traversal or picks
one of its kernels) or render enough samples for it (BDPT)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", ["JOB_COUNT_TRAVERSAL", "JOB_SIMPLE_EXTEND"])
def test_the_wavefront_reports_a_bound(ctx, flags):
    import gprt
    from gprt import capi, scenes
    g = gprt.GpuScene(ctx, scenes.icosphere_scene(level=4, width=40).to_desc(), test_stack_cap=True)
    r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=2, max_passes=1, seed=1,
                                                            flags=getattr(capi, flags)))
    with pytest.raises(capi.GprtError) as e:
        r.render_pass(1)
    assert e.value.code == capi.GPRT_E_BOUND
    r.close()
    g.close()


def test_the_bdpt_wavefront_reports_a_bound(ctx):
    import torch
    import gprt
    from gprt import capi, scenes
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    width = int((sms * 1024) ** 0.5) + 8  # one chunk of all pixels takes the wavefront
    g = gprt.GpuScene(ctx, scenes.icosphere_scene(level=4, width=width).to_desc(), test_stack_cap=True)
    r = gprt.ProgressiveRaytracer(g, gprt.ProgressiveConfig(max_samples_per_pixel=1, max_passes=1, seed=1),
                                  gprt.BDPTIntegrator())
    with pytest.raises(capi.GprtError) as e:
        r.render_pass(1)
    assert e.value.code == capi.GPRT_E_BOUND
    r.close()
    g.close()
