"""Ray groups (trace_group: eight or sixteen samples of a ray side by side in a warp) at the image
sizes where CTA shape and group size change and at sizes that leave partial tiles.

Image, sample counts and adjoint tape must not depend on which lanes a pixel falls to: the same
pixels rendered as a corner of a larger image (another CTA shape and group size) are equal bit for bit,
because a pixel's ray is formed from its own coordinates alone (orthographic view, spacing a power
of two) and each sample's arithmetic runs in one lane in the same order."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


def frame(ctx, vid, p, w, h):
    """(image, samples) of the [0, w/1024] x [0, h/1024] corner seen along +z, one pixel per 1/1024."""
    import torch

    ctx.set_params(p)
    ctx.set_view(wl.ortho_view(center=(w / 2048, h / 2048, 0.0), right=(w / 2048, 0, 0), up=(0, h / 2048, 0)))
    out = torch.zeros(h, w, 4, device="cuda")
    smp = torch.zeros(h, w, dtype=torch.int32, device="cuda")
    ctx.render_device(vid, out.data_ptr(), w, h, d_samples=smp.data_ptr())
    torch.cuda.synchronize()
    return out.cpu().numpy(), smp.cpu().numpy()


@pytest.mark.parametrize("integ", [capi.EULER, capi.HEUN, capi.RK4])
@pytest.mark.parametrize("lit", [False, True])
def test_pixels_do_not_depend_on_the_grid(ctx, integ, lit):
    rng = np.random.default_rng(7)
    vid = ctx.upload_field(wl.vortex_field(24, seed=3), storage="f16")
    ctx.upload_noise(rng.integers(0, 256, (20, 24, 28)).astype(np.uint8),
                     capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    rgba, op = wl.random_tf(5)
    ctx.set_tf(rgba, op)
    p = capi.params_default()
    p.integrator, p.steps_backward, p.steps_forward = integ, 3, 5
    p.step_size_vol = 1.0 / 32
    p.illum = capi.ILLUM_GRADIENT if lit else capi.ILLUM_NONE
    big, sbig = frame(ctx, vid, p, 1024, 1024)
    assert sbig.max() > 16
    for w, h in ((1, 1), (3, 2), (64, 31), (65, 57), (129, 130), (511, 3), (300, 258), (512, 512)):
        img, smp = frame(ctx, vid, p, w, h)
        np.testing.assert_array_equal(smp, sbig[:h, :w])
        np.testing.assert_array_equal(img, big[:h, :w])


@pytest.mark.parametrize("num_iterations", [1, 2, 3, 5])
def test_sample_bound_ends_rays_inside_a_group(ctx, num_iterations):
    """numIterations^2 samples at most: 1, 4, 9 and 25, inside and across groups of eight."""
    vid = ctx.upload_field(wl.abc_field(16))
    ctx.upload_noise(wl.dense_noise(16, seed=2))
    p = capi.params_default()
    p.num_iterations, p.alpha_threshold = num_iterations, 2.0
    p.steps_backward = p.steps_forward = 2
    p.step_size_vol = 1.0 / 64
    _, smp = frame(ctx, vid, p, 40, 24)
    np.testing.assert_array_equal(smp, min(num_iterations ** 2, 65))
