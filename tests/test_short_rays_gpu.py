"""Frames whose rays may end early or are short (launch_one): the first samples of each ray are taken one lane to
a ray, the rest in groups, or whole frames one lane to a ray.  The split depends on the frame's size, so
the pixels of a small frame, which is never split, must be those of a large one's corner, bit for bit, with
their sample counts; the adjoint of a split recording is the sum of its parts'."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


def transfer(kind):
    i = np.arange(256, dtype=np.float32)
    if kind == "opaque":
        return np.ones((256, 4), np.float32), np.ones(256, np.float32)
    alpha = (i > {"near": 150, "deep": 180}[kind]).astype(np.float32)
    return np.stack([i / 255] * 3 + [alpha], 1).astype(np.float32), np.linspace(0.2, 1, 256).astype(np.float32)


def frame(ctx, vid, p, w, h, tilt, x0=0, y0=0):
    """(image, samples, rays) of the w x h pixels from (x0, y0) on, one per 1/1024."""
    import torch

    ctx.set_params(p)
    ctx.set_view(wl.ortho_view(center=((x0 + w / 2) / 1024, (y0 + h / 2) / 1024, 0.0), right=(w / 2048, 0, 0), up=(0, h / 2048, 0),
                               direction=(tilt, 0.0, 1.0)))
    out = torch.full((h, w, 4), 7.0, device="cuda")  # whatever a pixel held before
    smp = torch.full((h, w), -1, dtype=torch.int32, device="cuda")
    ctx.render_device(vid, out.data_ptr(), w, h, d_samples=smp.data_ptr())
    torch.cuda.synchronize()
    st = ctx.stats()
    assert st.samples == int(smp.sum())
    return out.cpu().numpy(), smp.cpu().numpy(), st.rays


def same(ctx, vid, p, tilt=0.0):
    big, sbig, rays = frame(ctx, vid, p, 1024, 768, tilt)
    for x0, y0, w, h in ((0, 0, 150, 160), (512, 300, 160, 150), (850, 600, 171, 165), (300, 70, 64, 31)):
        img, smp, _ = frame(ctx, vid, p, w, h, tilt, x0, y0)
        np.testing.assert_array_equal(smp, sbig[y0:y0 + h, x0:x0 + w])
        np.testing.assert_array_equal(img, big[y0:y0 + h, x0:x0 + w])
    mid, smid, _ = frame(ctx, vid, p, 400, 330, tilt)  # another length of the first part
    np.testing.assert_array_equal(smid, sbig[:330, :400])
    np.testing.assert_array_equal(mid, big[:330, :400])
    return sbig, rays


def params(integ=capi.HEUN, lit=False):
    p = capi.params_default()
    p.integrator, p.steps_backward, p.steps_forward = integ, 3, 4
    p.step_size_vol, p.tf_index = 1.0 / 64, capi.TF_INDEX_MAGNITUDE
    p.illum = capi.ILLUM_GRADIENT if lit else capi.ILLUM_NONE
    return p


@pytest.mark.parametrize("tf", ["opaque", "near", "deep"])
@pytest.mark.parametrize("lit", [False, True])
@pytest.mark.parametrize("storage,integ", [("f16", capi.HEUN), ("f32", capi.HEUN), ("u8", capi.EULER), ("f16", capi.RK4)])
def test_early_ending_rays(ctx, tf, lit, storage, integ):
    vid = ctx.upload_field(wl.vortex_field(24, seed=3), storage=storage)
    ctx.upload_noise(wl.dense_noise(20, seed=8), capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    ctx.set_tf(*transfer(tf))
    p = params(integ, lit)
    p.alpha_threshold = 0.95 if tf == "opaque" else 0.3
    smp, rays = same(ctx, vid, p, tilt=0.25)
    assert rays == np.count_nonzero(smp)
    if tf == "opaque":
        assert smp.max() == 1
    else:
        assert len(np.unique(smp)) > 3 and (smp.max() > 32 if tf == "deep" else smp.max() <= 32)


@pytest.mark.parametrize("num_iterations", [1, 2, 3, 4, 5])
def test_sample_bound_around_the_first_part(ctx, num_iterations):
    """1, 4, 9, 16 and 25 samples at most: within the first part, at its end and beyond."""
    vid = ctx.upload_field(wl.abc_field(16))
    ctx.upload_noise(wl.dense_noise(16, seed=2))
    ctx.set_tf(*transfer("opaque"))
    p = params()
    p.num_iterations, p.alpha_threshold = num_iterations, 0.9999
    rgba, op = transfer("opaque")
    rgba[:128, 3] = 0.1  # rays may end, most do not
    ctx.set_tf(rgba, op)
    smp, _ = same(ctx, vid, p)
    assert smp.max() == num_iterations ** 2


@pytest.mark.parametrize("lit", [False, True])
@pytest.mark.parametrize("nz", [1, 2, 5, 9, 14, 30])
def test_thin_volumes(ctx, lit, nz):
    """Rays of few samples: whole frames one lane to a ray, or in groups, by size and thickness."""
    vid = ctx.upload_field(wl.vortex_field((64, 48, nz), seed=3), storage="f16")
    ctx.upload_noise(wl.dense_noise(20, seed=8), capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    ctx.set_tf(*wl.random_tf(5))
    p = params(lit=lit)
    p.quirks = 0
    p.step_size_vol = 1.0 / 64
    smp, _ = same(ctx, vid, p, tilt=0.1)
    assert 0 < smp.max() <= nz + 2


def gradients(ctx, vid, p, cot, x0=0, y0=0):
    """Adjoint of the recorded frame of the pixels that the cotangent holds, from (x0, y0) on."""
    import torch

    h, w = cot.shape[:2]
    p.record_tape = 1
    _, smp, _ = frame(ctx, vid, p, w, h, 0.0, x0, y0)
    got = [torch.zeros(k, device="cuda") for k in (1024, 256, p.steps_backward + p.steps_forward + 1)]
    ctx.render_adjoint(vid, cot.contiguous().data_ptr(), w, h, *(g.data_ptr() for g in got))
    torch.cuda.synchronize()
    assert (ctx.stats().check_flags or 0) == 0
    return [g.cpu().numpy().astype(np.float64) for g in got], smp


@pytest.mark.parametrize("integ", [capi.EULER, capi.HEUN, capi.RK4])
@pytest.mark.parametrize("lit", [False, True])
@pytest.mark.parametrize("case", ["short", "mixed", "thin"])
def test_adjoint_of_a_split_recording(ctx, lit, integ, case):
    """The gradients of a 520 x 480 frame are the sums of its twelve parts', none of which is split: rays that end at
    alpha 0.14 somewhere along the way, at 9 or 36 samples otherwise, and rays of two samples.  Tolerance:
    the sums' and the tap reductions' FP32 rounding."""
    import torch

    nz = 2 if case == "thin" else 16
    vid = ctx.upload_field(wl.vortex_field((16, 16, nz), seed=3), storage="f16")
    ctx.upload_noise(wl.dense_noise(20, seed=8), capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    i = np.arange(256, dtype=np.float32)
    ctx.set_tf(np.stack([i / 255] * 3 + [0.2 + 0 * i], 1), i / 255)
    p = params(integ, lit)
    p.quirks, p.gradient_scale = 0, 2.0
    p.step_size_vol, p.step_size_lic = (1.0 / 16, 0.02) if case == "thin" else (1.0 / 128, 0.02)
    p.num_iterations = 3 if case == "short" else 6
    p.alpha_threshold = 2.0 if case == "thin" else 0.14
    cot = torch.from_numpy(np.random.default_rng(3).standard_normal((480, 520, 4)).astype(np.float32)).cuda()
    got, smp = gradients(ctx, vid, p, cot)
    want = [np.zeros(g.shape) for g in got]
    for y0 in range(0, 480, 160):
        for x0 in range(0, 520, 130):
            part, spart = gradients(ctx, vid, p, cot[y0:y0 + 160, x0:x0 + 130], x0, y0)
            np.testing.assert_array_equal(spart, smp[y0:y0 + 160, x0:x0 + 130])
            for a, b in zip(want, part):
                a += b
    assert smp.max() <= {"short": 9, "mixed": 36, "thin": 4}[case] and (case == "thin" or len(np.unique(smp)) > 5)
    for g, r in zip(got, want):
        assert np.abs(r).max() > 0
        assert np.abs(g - r).max() <= 1e-5 * np.abs(r).max()


@pytest.mark.parametrize("integ,lit,ends,lb,lf", [(capi.RK4, False, True, 3, 4), (capi.RK4, True, True, 17, 5),
                                                  (capi.RK4, True, False, 2, 18), (capi.HEUN, True, True, 16, 17),
                                                  (capi.EULER, False, True, 0, 33)])
def test_adjoint_by_lane_per_ray(ctx, integ, lit, ends, lb, lf):
    """A 1000 x 980 frame's adjoint takes a lane per ray (RK4: two samples of it at a time), its quarters' groups
    of eight samples: rays of odd and even lengths within and across segments of 32 samples, streamlines around the
    16 steps of a block of tap sums."""
    import torch

    vid = ctx.upload_field(wl.vortex_field(16, seed=3), storage="f16")
    ctx.upload_noise(wl.dense_noise(20, seed=8), capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    i = np.arange(256, dtype=np.float32)
    ctx.set_tf(np.stack([i / 255] * 3 + [(0.2 if ends else 0.01) + 0 * i], 1), i / 255)
    p = params(integ, lit)
    p.quirks, p.gradient_scale, p.num_iterations = 0, 2.0, 6 if ends else 7
    p.steps_backward, p.steps_forward, p.step_size_vol, p.step_size_lic = lb, lf, 1.0 / 128, 0.02
    p.alpha_threshold = 0.14
    cot = torch.from_numpy(np.random.default_rng(3).standard_normal((980, 1000, 4)).astype(np.float32)).cuda()
    got, smp = gradients(ctx, vid, p, cot)
    assert (len(np.unique(smp)) > 5 and smp.max() == 36) if ends else np.all(smp == 49)
    # parts small enough for groups: below 16 times the resident warps where rays may end
    nx, ny = (2, 2) if integ == capi.RK4 else (5, 5)
    w, h = 1000 // nx, 980 // ny
    want = [np.zeros(g.shape) for g in got]
    for y0 in range(0, 980, h):
        for x0 in range(0, 1000, w):
            part, _ = gradients(ctx, vid, p, cot[y0:y0 + h, x0:x0 + w], x0, y0)
            for a, b in zip(want, part):
                a += b
    for g, r in zip(got, want):
        assert np.abs(r).max() > 0
        assert np.abs(g - r).max() <= 1e-5 * np.abs(r).max()
