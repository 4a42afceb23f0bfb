"""Texture copies of a field (surface writes; F32 texels as three arrays) hold its texels at every
voxel of odd, uneven and edge extents.

An orthographic direct-volume frame along z whose pixel centres are the voxel centres in x and y
and whose samples lie half-way between two slices (weights 0, 1 and 1/2, exact in the texture unit's
8-bit weights) reads every texel; it must be the GATHER frame up to the rounding of the filtered
value: FP32 texels to float rounding, the narrower ones to a half's 2^-11 per component, which the
alpha correction (exponent 128 * spacing, at most 128 / 5) and the front-to-back sum can scale by
that exponent."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "u8"])
@pytest.mark.parametrize("dims", [(1, 1, 5), (33, 2, 7), (5, 31, 64), (64, 64, 64), (257, 3, 9)])
def test_texture_copy_holds_every_texel(ctx, storage, dims):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx * 1000 + ny * 10 + nz)
    vid = ctx.upload_field(rng.standard_normal((nz, ny, nx, 3)).astype(np.float32), storage=storage)
    ctx.upload_noise(np.zeros((4, 4, 4), np.uint8))
    ext = np.array(dims, np.float64) / max(dims)
    p = capi.params_default()
    p.technique = capi.TECHNIQUE["volume"]
    p.step_size_vol = float(ext[2] / nz)
    p.alpha_threshold = 2.0
    ctx.set_view(wl.ortho_view(center=(ext[0] / 2, ext[1] / 2, 0.0), right=(ext[0] / 2, 0, 0), up=(0, ext[1] / 2, 0)))
    images = {}
    for sampler in ("gather", "hybrid"):
        p.sampler = capi.SAMPLER[sampler]
        ctx.set_params(p)
        images[sampler] = ctx.render(vid, nx, ny)
    assert float(images["gather"][..., 3].max()) > 0
    tol = (2e-6 if storage == "f32" else 2.0 ** -11) * max(1.0, 128.0 * p.step_size_vol)
    np.testing.assert_allclose(images["hybrid"], images["gather"], rtol=0, atol=tol)
