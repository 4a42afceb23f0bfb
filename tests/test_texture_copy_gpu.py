"""Texture copies of a field (surface writes; F32 texels as three arrays) hold its texels at every
voxel of odd, uneven and edge extents.

An orthographic direct-volume frame along z whose pixel centres are the voxel centres in x and y
and whose samples lie half-way between two slices (weights 0, 1 and 1/2, exact in the texture unit's
8-bit weights) reads every texel; it must be the frame of the exact means up to the rounding of the filtered
value: FP32 texels to float rounding, the narrower ones to a half's 2^-11 per component, which the
alpha correction (exponent 128 * spacing, at most 128 / 5) and the front-to-back sum can scale by
that exponent."""
import numpy as np
import pytest

from vectorvisualization_gb300 import capi, workloads as wl

pytestmark = pytest.mark.gpu


def half_slice_frame(t, tf, samples):
    """The frame in 64 bits: samples at z = 0, 1/nz, ..., each the mean of its two neighbouring
    slices, blended front to back."""
    nz = t.shape[0]
    dest = np.zeros(t.shape[1:3] + (4,))
    for k in range(samples):
        f = 0.5 * (t[max(k - 1, 0)] + t[min(k, nz - 1)])
        u = np.clip(f[..., 3] * 256 - 0.5, 0, 255)
        i = np.minimum(u.astype(int), 254)
        al = (tf[i, 3] * (i + 1 - u) + tf[i + 1, 3] * (u - i))[..., None]
        dest = np.clip(dest + (1 - dest[..., 3:]) * np.concatenate([f[..., :3] * al, al], -1), 0, 1)
    return dest


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
    p.sampler = capi.SAMPLER["hybrid"]
    ctx.set_params(p)
    ctx.set_view(wl.ortho_view(center=(ext[0] / 2, ext[1] / 2, 0.0), right=(ext[0] / 2, 0, 0), up=(0, ext[1] / 2, 0)))
    img = ctx.render(vid, nx, ny)
    samples = ctx.stats().samples // (nx * ny)  # a sample on the far face itself may be taken or not
    assert samples in (nz, nz + 1)
    ref = half_slice_frame(ctx.download_field(vid, dims, storage).astype(np.float64), ctx.get_tf()[0].astype(np.float64),
                           samples)
    assert float(ref[..., 3].max()) > 0
    tol = (2e-6 if storage == "f32" else 2.0 ** -11) * max(1.0, 128.0 * p.step_size_vol)
    np.testing.assert_allclose(img, ref, rtol=0, atol=tol)


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "u8"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (8, 4, 8), (9, 5, 7), (31, 33, 9), (33, 8, 17), (70, 3, 2)])
def test_update_writes_texels_and_arrays(ctx, storage, dims):
    """The update's encode writes texels and texture arrays in one kernel: the frame, and the texels
    read back, are those of a fresh upload bit for bit (32 x 8 x 8 voxel tiles and their remainders)."""
    nx, ny, nz = dims
    rng = np.random.default_rng(sum(dims))
    a, b = (rng.standard_normal((nz, ny, nx, 3)).astype(np.float32) for _ in range(2))
    ctx.upload_noise(rng.integers(0, 256, (8, 8, 8)).astype(np.uint8))
    p = capi.params_default()
    p.steps_backward = p.steps_forward = 4
    p.tf_index = capi.TF_INDEX_MAGNITUDE
    ctx.set_params(p)
    ext = np.array(dims, np.float64) / max(dims)
    ctx.set_view(wl.ortho_view(center=(ext[0] / 2, ext[1] / 2, 0.0), right=(ext[0] / 2, 0, 0), up=(0, ext[1] / 2, 0)))
    updated = ctx.upload_field(a, storage=storage)
    first = ctx.render(updated, 48, 40)
    ctx.update_field(updated, b)
    fresh = ctx.upload_field(b, storage=storage)
    img = ctx.render(updated, 48, 40)
    np.testing.assert_array_equal(img, ctx.render(fresh, 48, 40))
    np.testing.assert_array_equal(ctx.download_field(updated, dims, storage), ctx.download_field(fresh, dims, storage))
    if nx * ny * nz > 1:
        assert not np.array_equal(img, first)
