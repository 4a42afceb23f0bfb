"""The texel of a window sum from one reciprocal square root (pack_gradient in csrc/preprocess.cu), restated
in float32: wherever its margin lets the short form decide, its bytes are those of the reference's length, division
and double conversion (gradient.cpp:450-477), for every reciprocal square root that rsqrtf's bound of 2 ulp
allows, on sums whose components lie around each integer crossing."""
import numpy as np
import pytest

F32 = np.float32
MARGIN, CUT = F32(2e-4), F32(1e-8)


def squares(v):
    x, y, z = v.T
    return ((x * x).astype(F32) + (y * y).astype(F32)).astype(F32) + (z * z).astype(F32)


def exact(v):
    """Bytes of pack_gradient_exact: float length and quotients, the conversion in double."""
    ln = np.sqrt(squares(v)).astype(F32)[:, None]
    with np.errstate(all="ignore"):
        q = np.where(ln < F32(1e-5), F32(0), (v / ln).astype(F32))
    return np.trunc((q.astype(np.float64) + 1.0) / 2.0 * 255.0).astype(np.int64)


def short(v, ulps):
    """(bytes, whether the short form decides) with a reciprocal square root `ulps` off the rounded one."""
    s = squares(v)
    with np.errstate(all="ignore"):
        inv = (1.0 / np.sqrt(s.astype(np.float64))).astype(F32)
        inv = (inv.view(np.int32) + np.int32(ulps)).view(F32)
        # one rounding each: the product, and the FMA, whose product and sum are exact in double
        t = ((v * inv[:, None]).astype(F32).astype(np.float64) * 127.5 + 127.5).astype(F32)
        f = np.floor(t)
        r = t - f
        ok = (s > CUT) & (r > MARGIN).all(1) & (r < F32(1) - MARGIN).all(1)
    return np.where(ok[:, None], f, 0).astype(np.int64), ok


def sums(count, seed):
    """Window sums of length 1e-4 to 300, one component within 4e-4 byte steps of a crossing 1..254."""
    rng = np.random.default_rng(seed)
    k = np.tile(np.arange(1, 255), count)
    c = 2.0 * (k + rng.uniform(-4e-4, 4e-4, k.size)) / 255.0 - 1.0
    a = rng.uniform(0, 2 * np.pi, k.size)
    rest = np.sqrt(1 - c * c)
    v = np.stack([c, rest * np.cos(a), rest * np.sin(a)], 1)
    v = np.stack([np.roll(row, s) for row, s in zip(v, rng.integers(0, 3, k.size))])
    return (v * 10.0 ** rng.uniform(-4, 2.5, k.size)[:, None]).astype(F32)


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_short_form_agrees_around_every_crossing(ulps):
    v = sums(600, 7)
    got, ok = short(v, ulps)
    assert 0.2 < ok.mean() < 0.8  # both sides of the margin
    np.testing.assert_array_equal(got[ok], exact(v)[ok])


@pytest.mark.parametrize("ulps", [-2, 2])
def test_short_form_agrees_on_sums_of_byte_differences(ulps):
    """Sums of whole and half numbers, as unfiltered differences give them: axes, diagonals and equal
    components, whose unit vectors are the likeliest to lie on a crossing."""
    g = np.arange(-24, 25, dtype=np.float64) / 2
    v = np.stack(np.meshgrid(g, g, g), -1).reshape(-1, 3).astype(F32)
    got, ok = short(v, ulps)
    np.testing.assert_array_equal(got[ok], exact(v)[ok])
    assert not ok[(v == 0).all(1)].any()  # the zero sum takes the exact form
