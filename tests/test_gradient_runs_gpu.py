"""The one-pass noise gradients (noise_gradient_kernel) in the long slice runs of larger noises, against the
reference pipeline's CPU restatement, byte for byte: runs of 13, 25 and 64 slices, none a multiple of the
ring of three, each with a shorter last one."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi

pytestmark = pytest.mark.gpu


def run_length(nx, ny, nz):
    """Slices per CTA (launch_noise_gradients): 30 x 14 tiles over 152 * 12 CTAs, 8 to 64."""
    return min(max(-(-nz * -(-nx // 30) * -(-ny // 14) // (152 * 12)), 8), 64)


@pytest.mark.parametrize("mode", [capi.NOISE_GRAD_SOBEL, capi.NOISE_GRAD_CENTRAL])
@pytest.mark.parametrize("dims,run", [((300, 300, 100), 13), ((5, 2048, 310), 25), ((5, 2048, 794), 64)])
def test_long_runs_match_the_pipeline(vvlic_lib, oracle, mode, dims, run):
    import torch

    nx, ny, nz = dims
    assert run_length(*dims) == run and run % 3 and nz % run
    v = np.random.default_rng(run).integers(0, 256, (nz, ny, nx)).astype(np.uint8)
    d = torch.from_numpy(v).cuda()
    out = torch.zeros(nz, ny, nx, 4, dtype=torch.uint8, device="cuda")
    capi.noise_gradients_device(d.data_ptr(), dims, mode, out.data_ptr())
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.noise_gradients(v, mode))
