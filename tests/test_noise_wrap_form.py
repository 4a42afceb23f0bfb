"""The library's own choice of the noise cells' wrap form (csrc/noise_wrap.hpp), compiled with the host
compiler: the bound of a LIC volume's voxels and of a ray's start, the line between the forms, and that the
form chosen for a bound is exact for every coordinate within it.  On a GPU, a LIC-volume precompute and a
ray-cast on each side of the line against the FP64 oracle; the coordinates are dyadic (no
streamline step, orthographic rays), so FP32 and FP64 positions agree."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_noise_wrap import BITS, MAGIC, add_down, constants
from vectorvisualization_gb300 import capi, workloads as wl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FAR, MASK, MUL = 0, 1, 2
SOURCE = """
#include "noise_wrap.hpp"
extern "C" {
double ray_start(const float* e, const float* s, const float* t, double origin, double dir) {
  return vvlic::ray_start_bound(e, s, t, origin, dir);
}
double voxel_start(const float* s) { return vvlic::voxel_start_bound(s); }
int form(double start, double reach, const float* n, const float* g, const int* m) {
  return vvlic::choose_noise_wrap(start, reach, n, g, m);
}
}
"""


@pytest.fixture(scope="module")
def wrap(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("wrap")
    (d / "w.cpp").write_text(SOURCE)
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-shared", "-fPIC", "-I",
                        os.path.join(ROOT, "vectorvisualization_gb300", "csrc"), str(d / "w.cpp"), "-o", str(d / "w.so")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(d / "w.so"))
    lib.ray_start.restype = lib.voxel_start.restype = C.c_double
    lib.ray_start.argtypes = [C.c_void_p] * 3 + [C.c_double] * 2
    lib.form.argtypes = [C.c_double, C.c_double] + [C.c_void_p] * 3
    return lib


def f3(*v):
    return (C.c_float * 3)(*v)


def geometry(n, sd=(1.0, 1.0, 1.0)):
    """extent, scale, inverse scale of a volume (make_geometry)."""
    size = [a * b for a, b in zip(n, sd)]
    return ([s / max(size) for s in size], [max(n) / s for s in size], [s / max(n) for s in size])


def form_of(wrap, start, reach, freq, m):
    s = f3(*(freq * k for k in m))
    return wrap.form(start, reach, s, s, (C.c_int * 3)(*m))


# thin volumes, whose scale is large and whose inverse scale, the scaleVol of lit shaders, is small
@pytest.mark.parametrize("n,sd,m,freq", [((2048, 2048, 2), (1, 1, 1), (64, 64, 1000), 8.0),
                                         ((64, 64, 8), (1, 1, 2.0 ** -11), (20, 24, 60), 8.0),
                                         ((512, 512, 512), (1, 1, 0.001), (64, 64, 1000), 16.0)])
def test_lic_volume_of_a_thin_lit_volume_takes_the_general_form(wrap, n, sd, m, freq):
    ext, scale, inv = geometry(n, sd)
    largest = max(s * freq * k for s, k in zip(scale, m))
    assert largest > 1 << 21  # beyond the exact range of the multiply-high quotient
    assert form_of(wrap, wrap.voxel_start(f3(*scale)), 0.3, freq, m) == FAR
    # the rays of its lit frames stay near: their scaleVol is the inverse scale
    tex = [a * b for a, b in zip(ext, scale)]
    assert form_of(wrap, wrap.ray_start(f3(*ext), f3(*inv), f3(*tex), 2.0, 0.0), 0.3, freq, m) == MUL


def test_line_between_the_forms(wrap):
    limit = (1 << 19) - 4096
    for m, near in (((64, 64, 64), MASK), ((60, 64, 64), MUL), ((64, 60, 2), MUL)):
        for k in (0, 1):
            freq = (limit - 1) / 1.01 / 64
            assert form_of(wrap, 1.0 - k, float(k), 0.999999 * freq, m) == near
            assert form_of(wrap, 1.0 - k, float(k), 1.000001 * freq, m) == FAR
            assert form_of(wrap, 1.0 - k, float(k), -1.000001 * freq, m) == FAR
    for bad in (float("nan"), float("inf")):
        assert form_of(wrap, bad, 0.0, 1.0, (64, 64, 64)) == FAR
        assert form_of(wrap, 0.0, bad, 1.0, (64, 64, 64)) == FAR
        assert form_of(wrap, wrap.voxel_start(f3(1.0, bad, 1.0)), 0.0, 1.0, (64, 64, 64)) == FAR
        assert form_of(wrap, wrap.ray_start(f3(1, 1, 1), f3(1, 1, 1), f3(1, bad, 1), 1.0, 0.0), 0.0, 1.0, (64, 64, 64)) == FAR
        assert wrap.form(1.0, 0.0, f3(64, bad, 64), f3(64, 64, 64), (C.c_int * 3)(64, 64, 64)) == FAR


def entry(o, d, ext, clamp):
    """Start of a ray as the kernels form it (ray_interval, ray_setup), in FP32."""
    F = np.float32
    with np.errstate(all="ignore"):
        tn, tf = F(-np.inf), F(np.inf)
        for i in range(3):
            if d[i] == 0:
                if o[i] < 0 or o[i] > ext[i]:
                    return None
                continue
            inv = F(1) / d[i]
            t0, t1 = (F(0) - o[i]) * inv, (ext[i] - o[i]) * inv
            tn, tf = np.fmax(tn, np.fmin(t0, t1)), np.fmin(tf, np.fmax(t0, t1))
        if not tn < tf or (clamp and not tf > 0):
            return None
        if clamp:
            tn = np.fmax(tn, F(0))
        return o + tn * d


def test_ray_starts_stay_within_their_bound(wrap):
    """Directions down to denormals, alone and beside large components, and origins up to 1e30 away:
    a ray's first position is within the bound, or the bound is infinite."""
    rng = np.random.default_rng(9)
    F = np.float32
    ext = np.array([1.0, 0.25, 0.5], F)
    one = f3(1, 1, 1)
    unbounded = finite = outside = 0
    for k in range(40000):
        d = (rng.standard_normal(3) * 10.0 ** rng.uniform(-45, 3, 3)).astype(F)
        if k % 2:
            d[rng.integers(0, 3, 2)] = 0
        if k % 3 == 0:
            d = rng.standard_normal(3).astype(F)
        if not np.any(d):
            continue
        if k % 5 == 0:  # a camera far away, aimed at the box
            t = 10.0 ** rng.uniform(0, 30)
            o = (rng.random(3) * ext - t * d.astype(np.float64)).astype(F)
        else:
            o = (rng.uniform(-0.2, 1.2, 3) * ext).astype(F)
        if not np.all(np.isfinite(o)):
            continue
        clamp = k % 7 == 0 and float(np.abs(d).max()) >= 0.5
        pos = entry(o, d, ext, clamp)
        if pos is None:
            continue
        bound = wrap.ray_start(f3(*ext), one, one, float(np.abs(o).max()), 0.0 if clamp else float(np.abs(d).max()))
        if np.isinf(bound):
            unbounded += 1
            continue
        finite += 1
        largest = float(np.nanmax(np.abs(pos))) if not np.all(np.isnan(pos)) else 0.0
        outside += largest > 1.0
        assert largest <= bound, (o, d, pos, bound)
    assert unbounded > 100 and finite > 5000 and outside > 100
    # the view that no bound holds for: a denormal direction from inside the box
    assert np.isinf(entry(np.array([0.5, 0.1, 0.2], F), np.array([0, 0, -1e-40], F), ext, False)[2])
    assert wrap.ray_start(f3(*ext), one, one, 0.5, 1e-40) == float("inf")
    assert form_of(wrap, wrap.ray_start(f3(*ext), one, one, 0.5, 1e-40), 0.0, 1.0, (60, 60, 60)) == FAR
    assert form_of(wrap, wrap.ray_start(f3(*ext), one, one, 1e12, 1.0), 0.0, 1.0, (60, 60, 60)) == FAR


def test_chosen_form_is_exact_within_its_bound(wrap):
    """Whatever the form, the cell it reads at any coordinate up to the bound is the floored remainder."""
    rng = np.random.default_rng(5)
    near = 0
    for _ in range(400):
        m = [int(v) for v in rng.integers(2, 2049, 3)]
        if rng.random() < 0.3:
            m = [1 << int(v) for v in rng.integers(1, 12, 3)]
        freq, start, reach = (float(np.float32(2.0 ** v)) for v in rng.uniform(-4, 12, 3))
        form = form_of(wrap, start, reach, freq, m)
        if form == FAR:
            continue
        near += 1
        for k in m:
            u = np.concatenate([[-1.0, 1.0], rng.uniform(-1, 1, 50)]) * (start + reach) * freq * k - 0.5
            u = u.astype(np.float32)
            clamp, off, mul = constants(k)
            u = np.maximum(u, np.float32(clamp))
            t = add_down(u)
            np.testing.assert_array_equal(t - MAGIC, np.floor(u))
            want = np.mod(np.floor(u).astype(np.int64), k)
            bits = t.view(np.uint32)
            if form == MASK:
                np.testing.assert_array_equal(bits & np.uint32(k - 1), want)
            else:
                b = (bits - BITS + np.uint32(off)).astype(np.uint64)
                np.testing.assert_array_equal(b - ((b * np.uint64(mul)) >> np.uint64(32)) * np.uint64(k), want)
    assert near > 50


def test_single_texels_are_two_cells(tmp_path, wrap):
    """Extents of one: both cells hold the texel, so every form reads it; the other extents are their own."""
    src = SOURCE + 'extern "C" int cells(int m) { return vvlic::noise_cell_extent(m); }'
    (tmp_path / "c.cpp").write_text(src)
    subprocess.run([shutil.which("g++") or shutil.which("c++"), "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "vectorvisualization_gb300", "csrc"), str(tmp_path / "c.cpp"), "-o",
                    str(tmp_path / "c.so")], check=True)
    cells = C.CDLL(str(tmp_path / "c.so")).cells
    assert [cells(m) for m in (1, 2, 3, 2048)] == [2, 2, 3, 2048]
    for m in ((200, 150, 1), (1, 1, 3), (1, 64, 64), (1, 1, 1)):
        form = form_of(wrap, 1.0, 0.5, 2.0, [cells(k) for k in m])
        assert form == (MASK if all(k & (k - 1) == 0 for k in m) else MUL)


# ------------------------------------------------------------------------------------------
# on a GPU
# ------------------------------------------------------------------------------------------
def still(ctx, oracle, n, sd, m, freq, sampler, lit):
    """A scene whose streamlines do not move: every tap reads the noise at its sample's position."""
    w = wl.c1(size=8, image=8)
    w.field, w.noise = wl.vortex_field(n, seed=5), wl.dense_noise(8, seed=6)
    w.noise = np.random.default_rng(7).integers(0, 256, (m[2], m[1], m[0])).astype(np.uint8)
    p = w.params
    p.integrator, p.steps_backward, p.steps_forward = capi.EULER, 2, 3
    p.step_size_lic, p.freq_scale, p.step_size_vol, p.gradient_scale = 0.0, freq, 1.0 / 64, 2.0
    p.sampler = capi.SAMPLER[sampler]
    noise = w.noise
    if lit:
        p.illum, w.noise_mode = capi.ILLUM_GRADIENT, capi.NOISE_GRAD_CENTRAL
        noise = oracle.noise_gradients(w.noise, w.noise_mode)
    sc = oracle.Scene(oracle.encode_field(w.field), noise, w.tf_rgba, w.tf_opac, filter_table=w.filter_table,
                      slice_dist=sd)
    wl.setup_context(ctx, w)
    return w, sc, ctx.upload_field(w.field, slice_dist=sd, storage="f32")


@pytest.mark.gpu
@pytest.mark.parametrize("sampler,tol", [("cell", 2e-6), ("hybrid", 1e-4)])
@pytest.mark.parametrize("lit", [False, True])
@pytest.mark.parametrize("sd,m,freq", [(2.0 ** -11, (20, 24, 60), 8.0), (2.0 ** -4, (20, 24, 60), 8.0),
                                       (2.0 ** -11, (16, 32, 64), 8.0), (1.0, (20, 24, 60), 1.0)])
def test_lic_volume_on_each_side_of_the_line(ctx, oracle, sampler, tol, lit, sd, m, freq):
    """Noise coordinates up to 7.4 million, 57 thousand, 7.9 million (powers of two) and 480.  Tolerance:
    eighteen FP32 roundings (cell), 0.011 of a noise step (hybrid)."""
    n = (64, 32, 8)
    w, sc, vid = still(ctx, oracle, n, (1.0, 1.0, sd), m, freq, sampler, lit)
    dims = (32, 16, 8)
    ctx.set_params(w.params)
    ctx.compute_lic_volume(vid, dims)
    got, ref = ctx.download_lic_volume(vid, dims), sc.lic_volume(w.params, dims)
    assert float(np.ptp(ref)) > 0.1 * float(np.abs(ref).max())
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("sampler", ["cell", "hybrid"])
@pytest.mark.parametrize("lit", [False, True])
@pytest.mark.parametrize("m,freq", [((60, 30, 60), 8192.0), ((60, 30, 60), 8704.0), ((64, 32, 64), 7936.0),
                                    ((64, 32, 64), 8192.0)])
def test_frame_on_each_side_of_the_line(ctx, oracle, sampler, lit, m, freq):
    w, sc, vid = still(ctx, oracle, (16, 16, 16), (1.0, 1.0, 1.0), m, freq, sampler, lit)
    view = wl.ortho_view()
    ctx.set_params(w.params)
    ctx.set_view(view)
    img = ctx.render(vid, 32, 16)
    ref, smp = sc.render(w.params, view, 32, 16)
    assert float(ref[..., :3].max()) > 0.01 and abs(int(ctx.stats().samples) - int(smp.sum())) <= 0.01 * smp.sum() + 2
    assert float(np.sqrt(np.mean((img.astype(np.float64) - ref) ** 2))) <= 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("technique", ["raycast", "slicing"])
@pytest.mark.parametrize("view", [wl.ortho_view(direction=(0.0, 0.0, -1e-40)), wl.ortho_view(direction=(1e-42, 0.0, 1e-40)),
                                  wl.perspective_view(distance=1.5e8, fovy=4e-7),
                                  wl.ortho_view(center=(0.5 - 1e5, 0.5 - 2e5, 0.5 - 3e5), direction=(0.1, 0.2, 0.3))])
def test_views_without_a_bound(ctx, oracle, technique, view):
    """Directions of denormal components (rays that begin at infinity) and cameras so far away that rays begin
    outside the box: the cells read what the general gather reads."""
    w, _, vid = still(ctx, oracle, (16, 16, 16), (1.0, 1.0, 1.0), (60, 30, 60), 4096.0, "cell", False)
    imgs = []
    for sampler in ("cell", "gather"):
        p = w.params
        p.sampler, p.technique, p.num_iterations = capi.SAMPLER[sampler], capi.TECHNIQUE[technique], 16
        ctx.set_params(p)
        ctx.set_view(view)
        imgs.append(ctx.render(vid, 40, 24))
        assert technique == "slicing" or view.projection == capi.PERSPECTIVE or ctx.stats().samples > 0
    np.testing.assert_allclose(imgs[0], imgs[1], rtol=0, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [(20, 15, 1), (1, 15, 20), (12, 1, 1), (1, 1, 1), (16, 32, 1), (1, 7, 2)])
@pytest.mark.parametrize("freq", [1.0, -2.0, 65536.0])
def test_noise_of_a_single_texel_along_an_axis(ctx, m, freq):
    """CELL reads what GATHER reads, in the fast forms and (65536) the general one, also after the noise is
    replaced in place."""
    ctx.upload_field(wl.vortex_field(12, seed=3))
    w = wl.c1(size=12, image=8)
    vid = wl.setup_context(ctx, w)
    p = w.params
    p.steps_backward, p.steps_forward, p.freq_scale, p.step_size_lic = 3, 4, freq, 0.0
    ctx.set_view(wl.ortho_view())
    rng = np.random.default_rng(1)
    for _ in range(2):
        ctx.upload_noise(rng.integers(0, 256, m[::-1]).astype(np.uint8))
        imgs = []
        for sampler in ("cell", "gather"):
            p.sampler = capi.SAMPLER[sampler]
            ctx.set_params(p)
            imgs.append(ctx.render(vid, 33, 18))
        np.testing.assert_allclose(imgs[0], imgs[1], rtol=0, atol=2e-5)
