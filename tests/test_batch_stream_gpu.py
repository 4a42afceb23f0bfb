"""Streams a batch may not run on, and its use of those it may.  A first batch inside a caller's capture is
refused before it touches the capture, the context or the layouts."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


def scene(ctx, size, sampler="hybrid", count=3, storage="f16"):
    """(jobs, outputs, views) of a fresh volume and noise: no layout of theirs has been built yet."""
    import torch

    ctx.upload_noise(wl.dense_noise(16, seed=4))
    vid = ctx.upload_field(wl.vortex_field(12, seed=1), storage=storage)
    p = capi.params_default()
    p.steps_backward = p.steps_forward = 4
    p.sampler = capi.SAMPLER[sampler]
    ctx.set_params(p)
    ctx.set_filter_table(capi.make_filter_table("cos2", 64))
    outs = [torch.zeros(size, size, 4, device="cuda") for _ in range(count)]
    views = [wl.perspective_view(distance=2.0 + 0.3 * k) for k in range(count)]
    jobs = [capi.make_job(vid, o.data_ptr(), size, size, v, p, capi.make_filter_table("cos2", 64))
            for o, v in zip(outs, views)]
    return vid, jobs, outs, views


def check(ctx, vid, outs, views, size):
    for o, v in zip(outs, views):
        ctx.set_view(v)
        ref = ctx.render(vid, size, size)
        assert float(ref.max()) > 0
        np.testing.assert_array_equal(o.cpu().numpy(), ref)


@pytest.mark.parametrize("size", [16, 48])  # the persistent launch, jobs launched one by one
@pytest.mark.parametrize("sampler", ["hybrid", "texture", "cell"])
@pytest.mark.parametrize("mode", ["relaxed", "thread_local", "global"])
def test_first_batch_inside_a_capture(ctx, size, sampler, mode):
    import torch

    vid, jobs, outs, views = scene(ctx, size, sampler)
    stream = torch.cuda.Stream()
    word = torch.zeros(4, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode=mode)
        word.add_(1)
        with pytest.raises(capi.VVLICError) as e:
            ctx.batch_render(jobs, stream.cuda_stream)
        graph.capture_end()  # the capture goes on and ends cleanly
    assert e.value.status == capi.ERR_CUDA
    graph.replay()
    torch.cuda.synchronize()
    assert word.tolist() == [1.0] * 4
    assert all(float(o.abs().max()) == 0.0 for o in outs)
    ctx.batch_render(jobs, torch.cuda.Stream().cuda_stream)
    torch.cuda.synchronize()
    check(ctx, vid, outs, views, size)


@pytest.mark.parametrize("size", [16, 48])
def test_legacy_default_stream_is_refused(ctx, size):
    import torch

    vid, jobs, outs, views = scene(ctx, size)
    for _ in range(2):  # also once the shape's launch sequence exists
        with pytest.raises(capi.VVLICError) as e:
            ctx.batch_render(jobs, 1)  # cudaStreamLegacy
        assert e.value.status == capi.ERR_CUDA
        assert all(float(o.abs().max()) == 0.0 for o in outs)
        ctx.batch_render(jobs, torch.cuda.Stream().cuda_stream)
        torch.cuda.synchronize()
        check(ctx, vid, outs, views, size)
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()


def test_batch_keeps_its_streams_priority(ctx, vvlic_lib):
    """Jobs launched one by one on a high-priority stream, all eight of them, overtake a long frame of another
    context on a stream of default priority.  (A ninth job would queue behind the first of its side stream, and
    with the default of eight hardware queues that wait can hold up an unrelated stream's.)"""
    import torch

    vid, jobs, outs, views = scene(ctx, 64, count=8)
    high = torch.cuda.Stream(priority=-1)
    low = torch.cuda.Stream(priority=0)
    ctx.batch_render(jobs, low.cuda_stream)  # layouts, and streams of the other priority
    ctx.batch_render(jobs, high.cuda_stream)
    torch.cuda.synchronize()
    check(ctx, vid, outs, views, 64)
    with capi.Context(0) as other:
        other.upload_noise(wl.dense_noise(64, seed=4), capi.NOISE_GRAD_CENTRAL)
        big = other.upload_field(wl.vortex_field(64, seed=1), storage="f16")
        p = capi.params_default()
        p.integrator, p.illum, p.step_size_vol = capi.RK4, capi.ILLUM_GRADIENT, 1.0 / 512
        p.steps_backward = p.steps_forward = 60
        other.set_params(p)
        other.set_view(wl.perspective_view(distance=2.2))
        img = torch.empty(1024, 1024, 4, device="cuda")
        other.render_device(big, img.data_ptr(), 64, 64, stream=low.cuda_stream)
        torch.cuda.synchronize()
        done = torch.cuda.Event()
        other.render_device(big, img.data_ptr(), 1024, 1024, stream=low.cuda_stream)
        done.record(low)
        ctx.batch_render(jobs, high.cuda_stream)
        high.synchronize()
        assert not done.query()
        torch.cuda.synchronize()
