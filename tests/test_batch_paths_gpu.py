"""Both ways a batch runs (one persistent launch below a mean of 30 x 30 pixels, jobs launched one by
one from there on) at the line between them and with mixed sizes: every image is that of the job
rendered alone, bit for bit, and the totals are the jobs' sums."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(30, 30)], [(31, 30)] * 2, [(32, 32)] * 9, [(1, 1), (3, 2), (16, 9), (40, 20)],
                                   [(5, 3), (130, 70), (64, 64)], [(24, 20)] * 40])
@pytest.mark.parametrize("illum", [capi.ILLUM_NONE, capi.ILLUM_GRADIENT])
def test_batch_images_and_totals(ctx, sizes, illum):
    import torch

    ctx.upload_noise(wl.dense_noise(16, seed=4), capi.NOISE_GRAD_CENTRAL)
    vids = [ctx.upload_field(wl.vortex_field(n, seed=n), storage="f16") for n in (12, 17)]
    table = capi.make_filter_table("cos2", 64)
    ctx.set_filter_table(table)
    jobs, outs, alone, totals = [], [], [], np.zeros(3, np.int64)
    for k, (w, h) in enumerate(sizes):
        p = capi.params_default()
        p.steps_backward, p.steps_forward, p.illum = 3 + k % 5, 4, illum
        p.tf_index = capi.TF_INDEX_MAGNITUDE
        view = wl.perspective_view(wl.quat_axis_angle((1, 1, 0), 20.0 * k), distance=2.2)
        out = torch.zeros(h, w, 4, device="cuda")
        jobs.append(capi.make_job(vids[k % 2], out.data_ptr(), w, h, view, p, table))
        outs.append(out)
        ctx.set_params(p)
        ctx.set_view(view)
        alone.append(ctx.render(vids[k % 2], w, h))
        st = ctx.stats()
        totals += (st.samples, st.rays, st.sample_steps)
    stream = torch.cuda.Stream()
    for _ in range(2):  # the second call replays or relaunches
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        ctx.batch_render(jobs, stream.cuda_stream)
        stream.synchronize()
        for out, ref in zip(outs, alone):
            np.testing.assert_array_equal(out.cpu().numpy(), ref)
        st = ctx.stats()
        assert (st.samples, st.rays, st.sample_steps) == tuple(totals)


def test_batch_in_a_capture_is_refused(ctx):
    """Jobs launched one by one on a stream the caller is capturing are an error that leaves the capture
    as it was, and the next batch renders."""
    import torch

    size = 48

    ctx.upload_noise(wl.dense_noise(16, seed=4))
    vid = ctx.upload_field(wl.vortex_field(12, seed=1), storage="f16")
    p = capi.params_default()
    p.steps_backward = p.steps_forward = 4
    table = capi.make_filter_table("cos2", 64)
    outs = [torch.zeros(size, size, 4, device="cuda") for _ in range(2)]
    jobs = [capi.make_job(vid, o.data_ptr(), size, size, wl.perspective_view(distance=2.0 + k), p, table)
            for k, o in enumerate(outs)]
    stream = torch.cuda.Stream()
    ctx.batch_render(jobs, stream.cuda_stream)
    stream.synchronize()
    first = [o.cpu().numpy() for o in outs]
    scratch = torch.zeros(4, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        scratch.add_(1)
        with pytest.raises(capi.VVLICError):
            ctx.batch_render(jobs, stream.cuda_stream)
        graph.capture_end()
    for o in outs:
        o.zero_()
    torch.cuda.synchronize()
    ctx.batch_render(jobs, torch.cuda.Stream().cuda_stream)
    torch.cuda.synchronize()
    for o, ref in zip(outs, first):
        np.testing.assert_array_equal(o.cpu().numpy(), ref)
