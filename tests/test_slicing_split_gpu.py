"""Slicing frames of thin volumes, of few planes and under opaque tables (launch_tech_one), at sizes on both sides of
the lines between groups of planes and a lane per pixel: pixels and sample counts do not depend on the split, bit for
bit, and totals are the sums."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


def transfer(kind):
    rgba, op = np.ones((256, 4), np.float32), np.ones(256, np.float32)
    i = np.arange(256)
    if kind == "half":
        rgba[:128, 3] = 0.06
    elif kind == "ramp":
        rgba[:, 3] = np.maximum(0, i - 20) / 255
        op[:] = 0.6
    elif kind == "bands":
        rgba[:, 3] = 0.3 * ((i // 16) % 2)
    return rgba, op


@pytest.mark.parametrize("planes", [1, 2, 8, 20, 60])
@pytest.mark.parametrize("kind", ["opaque", "half", "ramp", "bands"])
@pytest.mark.parametrize("lit,integ,storage", [(False, capi.HEUN, "f16"), (True, capi.RK4, "f32")])
def test_slices_do_not_depend_on_the_split(ctx, planes, kind, lit, integ, storage):
    import torch

    vid = ctx.upload_field(wl.vortex_field(24, seed=3), storage=storage)
    ctx.upload_noise(wl.dense_noise(20, seed=8), capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    ctx.set_tf(*transfer(kind))
    p = capi.params_default()
    p.technique, p.integrator, p.steps_backward, p.steps_forward = capi.TECHNIQUE["slicing"], integ, 3, 5
    p.step_size_vol = 1.0 / (planes - 0.5)
    p.illum = capi.ILLUM_GRADIENT if lit else capi.ILLUM_NONE
    ctx.set_params(p)

    def frame(w, h):
        ctx.set_view(wl.ortho_view(center=(w / 2048, h / 2048, 0.0), right=(w / 2048, 0, 0), up=(0, h / 2048, 0)))
        out = torch.full((h, w, 4), 7.0, device="cuda")
        smp = torch.full((h, w), -1, dtype=torch.int32, device="cuda")
        ctx.render_device(vid, out.data_ptr(), w, h, d_samples=smp.data_ptr())
        torch.cuda.synchronize()
        st = ctx.stats()
        assert st.samples == int(smp.sum()) and st.rays == w * h
        return out.cpu().numpy(), smp.cpu().numpy()

    big, sbig = frame(500, 450)
    assert big.min() >= 0 and sbig.max() <= planes
    for w, h in ((61, 57), (171, 170), (172, 171), (243, 240), (245, 242), (421, 417)):
        img, smp = frame(w, h)
        np.testing.assert_array_equal(smp, sbig[:h, :w])
        np.testing.assert_array_equal(img, big[:h, :w])
