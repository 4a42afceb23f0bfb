"""The adjoint's ray groups (eight samples of four rays in a warp) and block-wise tap sums at the
sizes where they can go wrong: rays that end inside a chunk of eight and a segment of 32, images that
leave partial 2x2-ray tiles, and streamline lengths around the 16 steps of a sum block, even and
uneven, images one tile past a strip of 64 pixels and past two, for every integrator, against the FP64 adjoint.  Exact sampler and a frame inside (0, 1), away
from the blend's clamp where an FP32 and an FP64 state may take different branches; the tolerances are
those of the adjoint parity tests (2e-3 of the largest gradient, 1e-2 lit)."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integ", [capi.EULER, capi.HEUN, capi.RK4])
@pytest.mark.parametrize("lit", [False, True])
@pytest.mark.parametrize("lb,lf,bound,w,h", [(1, 0, 1, 5, 3), (15, 16, 3, 7, 6), (16, 15, 4, 6, 5), (17, 33, 5, 5, 4),
                                             (0, 20, 6, 3, 3), (31, 32, 7, 4, 2), (2, 3, 2, 65, 3), (3, 2, 2, 131, 2)])
def test_adjoint_at_chunk_and_block_edges(ctx, oracle, integ, lit, lb, lf, bound, w, h):
    import torch

    wk = wl.c4(size=16, image=8, views=1)
    p = wk.params
    p.integrator, p.steps_backward, p.steps_forward = integ, lb, lf
    p.step_size_vol, p.step_size_lic = 1.0 / 128, 0.02
    p.num_iterations = bound  # rays of 1, 9, 16, 25, 36 and 49 samples, none near the box's far face
    p.sampler, p.record_tape = capi.SAMPLER["cell"], 1
    p.alpha_threshold = 2.0
    p.gradient_scale = 2.0
    wk.tf_rgba, wk.tf_opac = wk.tf_rgba * np.float32(0.25), wk.tf_opac * np.float32(0.25)
    if lit:
        p.illum, wk.noise_mode = capi.ILLUM_GRADIENT, capi.NOISE_GRAD_CENTRAL
    view = wl.ortho_view()
    wk.views = [view]
    vid = wl.setup_context(ctx, wk)
    img = torch.empty(h, w, 4, device="cuda")
    ctx.render_device(vid, img.data_ptr(), w, h)
    assert 0.0 < float(img.max()) < 1.0 and ctx.stats().samples == bound ** 2 * w * h
    cot = torch.from_numpy(np.random.default_rng(3).standard_normal((h, w, 4)).astype(np.float32)).cuda()
    got = [torch.zeros(k, device="cuda") for k in (1024, 256, lb + lf + 1)]
    ctx.render_adjoint(vid, cot.data_ptr(), w, h, *(g.data_ptr() for g in got))
    torch.cuda.synchronize()
    noise = oracle.noise_gradients(wk.noise, wk.noise_mode) if lit else wk.noise
    sc = oracle.Scene(oracle.encode_field(wk.field), noise, wk.tf_rgba, wk.tf_opac, filter_table=wk.filter_table)
    want = oracle.adjoint(sc, p, view, w, h, cot.cpu().numpy())
    for g, r in zip(got, want):
        r = np.asarray(r, np.float64).ravel()
        assert np.abs(g.cpu().numpy() - r).max() <= (1e-2 if lit else 2e-3) * np.abs(r).max()
