"""The slicing kernel's plane queue at its edges: fewer planes than a group of eight, whole groups, one
more, TFs that pass none, few, alternating and all of the planes, rays that turn opaque inside a
group, and image sizes that leave partial 2x2-ray tiles, against the FP64 oracle (RMSE <= 1e-3 and
sample counts within 1 % + 2, the bar of the technique tests: a plane on the box or the alpha gate
may fall to either side)."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes", [1, 3, 8, 9, 17, 40])
@pytest.mark.parametrize("gate", ["none", "few", "bands", "all", "opaque"])
def test_slicing_queue_edges(ctx, oracle, planes, gate):
    w = wl.c1(size=20, image=8)
    w.field = wl.vortex_field(20, seed=9)
    w.noise = wl.dense_noise(20, seed=91)
    p = w.params
    p.integrator, p.steps_backward, p.steps_forward = capi.HEUN, 3, 4
    p.technique, p.sampler = capi.TECHNIQUE["slicing"], capi.SAMPLER["cell"]
    p.step_size_vol = 1.0 / (planes - 0.5)  # a unit depth along z: `planes` slices
    i = np.arange(256)
    alpha = {"none": 0.0 * i, "few": 0.3 * (i > 200), "bands": 0.3 * ((i // 16) % 2), "all": 0.2 + 0.0 * i,
             "opaque": 0.9 + 0.0 * i}[gate]
    w.tf_rgba[:, 3] = alpha
    w.tf_opac[:] = np.maximum(w.tf_opac, 0.9 if gate == "opaque" else 0.3)
    noise = w.noise
    sc = oracle.Scene(oracle.encode_field(w.field), noise, w.tf_rgba, w.tf_opac, filter_table=w.filter_table)
    vid = wl.setup_context(ctx, w)
    view = wl.ortho_view()
    ctx.set_view(view)
    for size in ((1, 1), (7, 5), (33, 18)):
        img = ctx.render(vid, *size)
        ref, smp = sc.render(p, view, *size)
        assert float(np.sqrt(np.mean((img.astype(np.float64) - ref) ** 2))) <= 1e-3
        assert abs(int(ctx.stats().samples) - int(smp.sum())) <= 0.01 * smp.sum() + 2
        assert (gate == "none") == (smp.sum() == 0 and float(img.max()) == 0.0) or gate == "few"


@pytest.mark.parametrize("integ", [capi.EULER, capi.HEUN, capi.RK4])
@pytest.mark.parametrize("lit", [False, True])
def test_slices_do_not_depend_on_the_grid(ctx, integ, lit):
    """Groups of eight planes (small frames), of two (medium ones) and a lane per pixel (large ones) give a
    pixel the same value and count, bit for bit: the corner of a larger frame is the smaller frame."""
    import torch

    vid = ctx.upload_field(wl.vortex_field(24, seed=3), storage="f16")
    ctx.upload_noise(wl.dense_noise(20, seed=8), capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    ctx.set_tf(*wl.random_tf(5))
    p = capi.params_default()
    p.technique, p.integrator, p.steps_backward, p.steps_forward = capi.TECHNIQUE["slicing"], integ, 3, 5
    p.step_size_vol = 1.0 / 99.5  # 100 planes
    p.illum = capi.ILLUM_GRADIENT if lit else capi.ILLUM_NONE
    ctx.set_params(p)

    def frame(w, h):
        ctx.set_view(wl.ortho_view(center=(w / 2048, h / 2048, 0.0), right=(w / 2048, 0, 0), up=(0, h / 2048, 0)))
        out = torch.zeros(h, w, 4, device="cuda")
        smp = torch.zeros(h, w, dtype=torch.int32, device="cuda")
        ctx.render_device(vid, out.data_ptr(), w, h, d_samples=smp.data_ptr())
        torch.cuda.synchronize()
        return out.cpu().numpy(), smp.cpu().numpy()

    big, sbig = frame(1024, 1024)
    assert sbig.max() > 8
    for w, h in ((1, 1), (65, 57), (300, 258), (419, 418), (420, 421), (513, 509), (603, 604), (611, 605)):
        img, smp = frame(w, h)
        np.testing.assert_array_equal(smp, sbig[:h, :w])
        np.testing.assert_array_equal(img, big[:h, :w])
