"""LIC-volume frames with two and with four samples in flight (launch_tech_layout): opacities that no sample reads
change how many are, and no pixel or count, at every number of samples modulo both."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iterations", [1, 2, 3, 64])  # 1, 4 and 9 samples at most; all
@pytest.mark.parametrize("opacity", [0.02, 0.3, 0.8])  # rays that go on, and that end inside a batch
@pytest.mark.parametrize("storage", ["f16", "f32"])
def test_samples_in_flight_do_not_show(ctx, iterations, opacity, storage):
    import torch

    vid = ctx.upload_field(wl.vortex_field(20, seed=3), storage=storage)
    ctx.upload_noise((wl.dense_noise(20, seed=8) // 64).astype(np.uint8), capi.NOISE_SCALAR)  # intensities below 0.3
    p = capi.params_default()
    p.steps_backward = p.steps_forward = 4
    p.tf_index, p.step_size_vol, p.num_iterations = capi.TF_INDEX_MAGNITUDE, 1.0 / 20, iterations
    ctx.set_params(p)
    ctx.compute_lic_volume(vid, (20, 20, 20))
    p.technique = capi.TECHNIQUE["licvolume"]
    ctx.set_params(p)
    ctx.set_view(wl.ortho_view(direction=(0.2, 0.1, 1.0)))
    frames = []
    for unread in (opacity, 1.0):  # a share of 0, and of 0.53
        op = np.full(256, opacity, np.float32)
        op[120:] = unread
        ctx.set_tf(np.ones((256, 4), np.float32), op)
        out = torch.full((29, 37, 4), 7.0, device="cuda")
        smp = torch.full((29, 37), -1, dtype=torch.int32, device="cuda")
        ctx.render_device(vid, out.data_ptr(), 37, 29, d_samples=smp.data_ptr())
        torch.cuda.synchronize()
        assert ctx.stats().samples == int(smp.sum())
        frames.append((out.cpu().numpy(), smp.cpu().numpy()))
    np.testing.assert_array_equal(frames[0][1], frames[1][1])
    np.testing.assert_array_equal(frames[0][0], frames[1][0])
    assert frames[0][1].max() <= iterations ** 2
