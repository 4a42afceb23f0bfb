"""Batches whose rays end after a sample or two, or are no longer (expected_samples in batch.cu): the persistent launch
with a lane to a ray, also for jobs that would be launched one by one otherwise, at the sizes where the route changes,
under every tile width.  Every image is that of the job rendered alone, bit for bit, and the totals are the jobs' sums."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


def transfer(kind):
    rgba, op = np.ones((256, 4), np.float32), np.ones(256, np.float32)
    if kind != "opaque":
        rgba[:, 3] = 0.2
        rgba[:int(kind), 3] = 1.0  # so many of 256 alphas end a ray
    return rgba, op


# (alphas that end a ray, slices of the volume)
@pytest.mark.parametrize("kind,slices", [("opaque", 16), ("128", 16), ("127", 16), ("0", 1), ("0", 3)])
@pytest.mark.parametrize("sizes", [[(1, 1)], [(5, 3), (16, 9), (29, 30)], [(33, 31)] * 9, [(121, 121)], [(123, 119), (7, 130)]])
@pytest.mark.parametrize("illum,integ", [(capi.ILLUM_NONE, capi.HEUN), (capi.ILLUM_GRADIENT, capi.RK4)])
def test_brief_batches(ctx, kind, slices, sizes, illum, integ):
    import torch

    ctx.upload_noise(wl.dense_noise(16, seed=4), capi.NOISE_GRAD_CENTRAL)
    field = wl.vortex_field(16, seed=9)
    vid = ctx.upload_field(np.ascontiguousarray(field[:slices]), storage="f16")
    ctx.set_tf(*transfer(kind))
    table = capi.make_filter_table("cos2", 64)
    ctx.set_filter_table(table)
    jobs, outs = [], []
    for k, (w, h) in enumerate(sizes):
        p = capi.params_default()
        p.steps_backward, p.steps_forward, p.illum, p.integrator = 3 + k % 5, 4, illum, integ
        p.tf_index, p.step_size_vol = capi.TF_INDEX_MAGNITUDE, 1.0 / 16
        view = wl.perspective_view(wl.quat_axis_angle((1, 1, 0), 3.0 * k + 1.0), distance=2.2)
        outs.append(torch.zeros(h, w, 4, device="cuda"))
        jobs.append(capi.make_job(vid, outs[-1].data_ptr(), w, h, view, p, table))
    stream = torch.cuda.Stream()

    def check(sampler):
        alone, totals = [], np.zeros(3, np.int64)
        for job in jobs:
            p = capi.Params.from_buffer_copy(job.params)
            p.sampler = sampler
            ctx.set_params(p)
            ctx.set_view(job.view)
            alone.append(ctx.render(vid, job.w, job.h))
            st = ctx.stats()
            totals += (st.samples, st.rays, st.sample_steps)
        for out in outs:
            out.fill_(7.0)
        torch.cuda.synchronize()
        ctx.batch_render(jobs, stream.cuda_stream)
        stream.synchronize()
        for out, ref in zip(outs, alone):
            np.testing.assert_array_equal(out.cpu().numpy(), ref)
        st = ctx.stats()
        assert (st.samples, st.rays, st.sample_steps) == tuple(totals)

    check(jobs[0].params.sampler)
    ctx.set_tf(*transfer("0" if kind == "opaque" else "opaque"))  # the same shapes, another split of the work
    check(jobs[0].params.sampler)
    ctx.set_tf(*transfer(kind))
    check(ctx.batch_autotune(jobs, stream.cuda_stream)[1])  # every tile width, and the tuned one
