"""The one-pass noise gradients (noise_gradient_kernel) at the edges of its tiles and slice runs,
against the reference pipeline's CPU restatement, byte for byte: 30 x 14 output tiles, runs of 8 to
64 slices, extents below the smoothing window, and every border rule, in both modes and with
anisotropic slice distances."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 2), (3, 2, 5), (5, 5, 5), (30, 14, 8), (31, 15, 9), (29, 13, 7), (32, 16, 64), (33, 17, 65), (61, 29, 66),
        (100, 3, 2), (2, 40, 130)]


@pytest.mark.parametrize("mode", [capi.NOISE_GRAD_SOBEL, capi.NOISE_GRAD_CENTRAL])
@pytest.mark.parametrize("kind", ["dense", "sparse", "flat"])
def test_one_pass_gradients_match_the_pipeline(vvlic_lib, oracle, mode, kind):
    import torch

    rng = np.random.default_rng(11)
    for nx, ny, nz in DIMS:
        v = {"dense": rng.integers(0, 256, (nz, ny, nx)), "sparse": 255 * (rng.random((nz, ny, nx)) < 0.05),
             "flat": np.full((nz, ny, nx), 7)}[kind].astype(np.uint8)
        for sd in ((1.0, 1.0, 1.0), (1.0, 0.5, 3.0)):
            d = torch.from_numpy(v).cuda()
            out = torch.zeros(nz, ny, nx, 4, dtype=torch.uint8, device="cuda")
            capi.noise_gradients_device(d.data_ptr(), (nx, ny, nz), mode, out.data_ptr(), slice_dist=sd)
            want = oracle.noise_gradients(v, mode, slice_dist=sd)
            np.testing.assert_array_equal(out.cpu().numpy(), want, err_msg=f"{nx}x{ny}x{nz} {sd}")
