"""An FP32 volume's texture copy is three arrays: when memory ends between them, the render fails and leaves
nothing allocated, and succeeds once there is room."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


def test_failed_texture_copy_holds_no_memory(ctx):
    import torch

    n = 256  # arrays of 128, 64 and 64 MiB
    field = np.broadcast_to(np.float32([0.3, 0.4, 0.5]), (n, n, n, 3))
    vid = ctx.upload_field(field, storage="f32")
    ctx.upload_noise(np.zeros((8, 8, 8), np.uint8))
    ctx.set_view(wl.ortho_view())
    p = capi.params_default()
    p.technique, p.step_size_vol, p.sampler = capi.TECHNIQUE["volume"], 1.0 / 16, capi.SAMPLER["gather"]
    ctx.set_params(p)
    out = torch.empty(16, 16, 4, device="cuda")
    ctx.render_device(vid, out.data_ptr(), 16, 16)  # everything but the texture copy is in place
    want = out.clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    mib = 1 << 20
    hold = [torch.empty(torch.cuda.mem_get_info()[0] - 1024 * mib, dtype=torch.uint8, device="cuda")]
    while torch.cuda.mem_get_info()[0] > 200 * mib:  # room for the first array, not for all three
        hold.append(torch.empty(32 * mib, dtype=torch.uint8, device="cuda"))
    p.sampler = capi.SAMPLER["hybrid"]
    ctx.set_params(p)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        with pytest.raises(capi.VVLICError) as e:
            ctx.render_device(vid, out.data_ptr(), 16, 16)
        assert e.value.status == capi.ERR_OUT_OF_MEMORY
        assert free - torch.cuda.mem_get_info()[0] < 32 * mib
    hold.clear()
    torch.cuda.empty_cache()
    ctx.render_device(vid, out.data_ptr(), 16, 16)
    torch.cuda.synchronize()
    np.testing.assert_allclose(out.cpu().numpy(), want.cpu().numpy(), rtol=0, atol=1e-2)
