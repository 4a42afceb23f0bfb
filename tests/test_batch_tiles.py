"""The persistent batch launch at every tile width: the mapping of a tile's lanes to pixels (csrc/batch_tiles.hpp,
compiled with the host compiler) takes each pixel of an image once; on a GPU, small batches under the
autotuner, which renders every width, and replayed with changed views."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "batch_tiles.hpp"
extern "C" void pixels(int tw, int w, int h, int* count, int* outside) {
  const int th = 32 / tw, tx = (w + tw - 1) / tw, ty = (h + th - 1) / th;
  for (int tile = 0; tile < tx * ty; ++tile)
    for (int sub = 0; sub < 4; ++sub)
      for (int r = 0; r < 8; ++r) {
        const vvlic::BatchPixel p = vvlic::batch_pixel(tw, tile, tx, sub, r);
        if (p.x < 0 || p.y < 0 || p.x >= tx * tw || p.y >= ty * th) ++*outside;
        else if (p.x < w && p.y < h) ++count[p.y * w + p.x];
      }
}
"""


@pytest.mark.parametrize("tw", [4, 8, 16, 32])
def test_tiles_take_each_pixel_once(tmp_path, tw):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "vectorvisualization_gb300", "csrc"), str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t.so")], check=True)
    lib = C.CDLL(str(tmp_path / "t.so"))
    for w in (1, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 40):
        for h in (1, 2, 3, 4, 7, 8, 9, 21):
            count, outside = np.zeros((h, w), np.int32), C.c_int(0)
            lib.pixels(tw, w, h, count.ctypes.data_as(C.POINTER(C.c_int)), C.byref(outside))
            assert outside.value == 0
            np.testing.assert_array_equal(count, 1)


def small_jobs(ctx, sizes, illum=capi.ILLUM_NONE):
    import torch

    ctx.upload_noise(wl.dense_noise(16, seed=4), capi.NOISE_GRAD_CENTRAL)
    vids = [ctx.upload_field(wl.vortex_field(n, seed=n), storage="f16") for n in (12, 17)]
    table = capi.make_filter_table("cos2", 64)
    ctx.set_filter_table(table)
    jobs, outs = [], []
    for k, (w, h) in enumerate(sizes):
        p = capi.params_default()
        p.steps_backward, p.steps_forward, p.illum = 3 + k % 5, 4, illum
        view = wl.perspective_view(wl.quat_axis_angle((1, 1, 0), 20.0 * k), distance=2.2)
        outs.append(torch.zeros(h, w, 4, device="cuda"))
        jobs.append(capi.make_job(vids[k % 2], outs[-1].data_ptr(), w, h, view, p, table))
    return jobs, outs


def check(ctx, jobs, outs, sampler):
    for job, out in zip(jobs, outs):
        p = capi.Params.from_buffer_copy(job.params)
        p.sampler = sampler
        ctx.set_params(p)
        ctx.set_view(job.view)
        np.testing.assert_array_equal(out.cpu().numpy(), ctx.render(job.vol_id, job.w, job.h))


SIZES = [(1, 1), (5, 3), (24, 20), (17, 9), (33, 7), (3, 33), (40, 2), (16, 8)]


@pytest.mark.gpu
@pytest.mark.parametrize("illum", [capi.ILLUM_NONE, capi.ILLUM_GRADIENT])
def test_autotuned_small_batches(ctx, illum):
    """The autotuner's last render is the 32-pixel rows with the cell sampler; the batch then runs at the width
    it found, also after a batch of large jobs has been tuned."""
    import torch

    jobs, outs = small_jobs(ctx, SIZES, illum)
    stream = torch.cuda.Stream()
    tw, smp, ms = ctx.batch_autotune(jobs, stream.cuda_stream)
    stream.synchronize()
    assert tw in (4, 8, 16, 32) and ms > 0
    check(ctx, jobs, outs, capi.SAMPLER["cell"])
    for large in (False, True):
        if large:
            big, _ = small_jobs(ctx, [(64, 64)] * 2, illum)
            tw, smp, _ = ctx.batch_autotune(big, stream.cuda_stream)
            assert tw == 8
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        ctx.batch_render(jobs, stream.cuda_stream)
        stream.synchronize()
        check(ctx, jobs, outs, smp)


@pytest.mark.gpu
def test_small_batch_replay_follows_changed_views(ctx):
    import torch

    jobs, outs = small_jobs(ctx, [(24, 20)] * 7)
    stream = torch.cuda.Stream()
    rng = wl.SplitMix64(99)
    for _ in range(3):  # captured, then replayed
        ctx.batch_render(jobs, stream.cuda_stream)
        stream.synchronize()
        check(ctx, jobs, outs, jobs[0].params.sampler)
        for j in jobs:
            j.view = wl.random_view(rng)
