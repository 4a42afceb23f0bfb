// Render entry points: uniform derivation (Renderer::setRenderVolParams, renderer.cpp:925-996),
// lazy construction of the field/noise layouts the chosen sampler reads, and the launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <chrono>
#include <cstring>
#include <thread>

#include "../../include/vvlic.h"
#include "brick.cuh"
#include "vvlic_device.cuh"
#include "vvlic_host.hpp"
#include "vvlic_launch.hpp"

using namespace vvlic;

namespace {

vvlic_status ensure_cells(vvlic_ctx* c, Volume& v, cudaStream_t s) {
  if (v.d_cells) return VVLIC_OK;
  const size_t cells = (size_t)(v.n[0] + 1) * (v.n[1] + 1) * (v.n[2] + 1);
  const size_t bytes = cells * 8 * texel_bytes(v.storage);
  cudaError_t e = cudaMalloc(&v.d_cells, bytes);
  if (e != cudaSuccess) return cuda_fail(c, e, "cell layout allocation");
  v.cell_bytes = bytes;
  e = launch_build_field_cells(v.d_texels, v.n, v.storage, v.d_cells, s);
  if (e != cudaSuccess) return cuda_fail(c, e, "cell layout build");
  return VVLIC_OK;
}

vvlic_status ensure_noise_cells(vvlic_ctx* c, NoiseTex& n, cudaStream_t s) {
  if (n.d_cells) return VVLIC_OK;
  const int cells[3] = {noise_cell_extent(n.m[0]), noise_cell_extent(n.m[1]), noise_cell_extent(n.m[2])};
  const size_t bytes = noise_cell_count(cells) * 8 * n.ch;
  cudaError_t e = cudaMalloc(&n.d_cells, bytes);
  if (e != cudaSuccess) return cuda_fail(c, e, "noise cell allocation");
  e = launch_build_noise_cells(n.d_texels, n.m, n.ch, n.d_cells, s);
  if (e != cudaSuccess) return cuda_fail(c, e, "noise cell build");
  return VVLIC_OK;
}

FieldSurfaces surfaces(const Volume& v) {
  FieldSurfaces arr;
  arr.rgba = v.surf[0];
  arr.z = v.surf[1];
  arr.w = v.surf[2];
  return arr;
}

// Arrays, surfaces and textures of the texture copy.  128-bit texels filter at an eighth of the texture
// unit's rate, so F32 fields are held as a float2 array of (x, y) and two float arrays
// (Field<F32, kTexture>).
vvlic_status make_texture(vvlic_ctx* c, Volume& v) {
  const bool f32 = v.storage == VVLIC_STORAGE_F32, u8 = v.storage == VVLIC_STORAGE_UNORM8;
  const cudaChannelFormatDesc desc[3] = {f32 ? cudaCreateChannelDesc<float2>()
                                             : (u8 ? cudaCreateChannelDesc<uchar4>() : cudaCreateChannelDescHalf4()),
                                         cudaCreateChannelDesc<float>(), cudaCreateChannelDesc<float>()};
  const cudaExtent ext = make_cudaExtent(v.n[0], v.n[1], v.n[2]);
  for (int i = 0; i < (f32 ? 3 : 1); ++i) {
    cudaError_t e = cudaMalloc3DArray(&v.array[i], &desc[i], ext, cudaArraySurfaceLoadStore);
    if (e != cudaSuccess) return cuda_fail(c, e, "texture array allocation");
    cudaResourceDesc rd;
    std::memset(&rd, 0, sizeof rd);
    rd.resType = cudaResourceTypeArray;
    rd.res.array.array = v.array[i];
    e = cudaCreateSurfaceObject(&v.surf[i], &rd);
    if (e != cudaSuccess) return cuda_fail(c, e, "texture surface");
    cudaTextureDesc td;
    std::memset(&td, 0, sizeof td);
    td.addressMode[0] = td.addressMode[1] = td.addressMode[2] = cudaAddressModeClamp;  // CLAMP_TO_EDGE
    td.filterMode = cudaFilterModeLinear;
    td.readMode = u8 ? cudaReadModeNormalizedFloat : cudaReadModeElementType;
    td.normalizedCoords = 1;  // GL texture coordinates
    e = cudaCreateTextureObject(&v.tex[i], &rd, &td, nullptr);
    if (e != cudaSuccess) return cuda_fail(c, e, "texture object");
  }
  return VVLIC_OK;
}

vvlic_status ensure_texture(vvlic_ctx* c, Volume& v, cudaStream_t s) {
  if (v.array_bytes) return VVLIC_OK;
  vvlic_status st = make_texture(c, v);
  if (!st) {
    const cudaError_t e = launch_fill_arrays(v.d_texels, v.n, v.storage, surfaces(v), s);
    if (e != cudaSuccess) st = cuda_fail(c, e, "texture array fill");
  }
  if (st) {
    free_textures(v);  // nothing stays allocated behind a failed call
    return st;
  }
  v.array_bytes = (size_t)v.n[0] * v.n[1] * v.n[2] * texel_bytes(v.storage);
  return VVLIC_OK;
}

// Noise as an R8 / RGBA8 texture read as normalised float with WRAP addressing (GL REPEAT).
vvlic_status copy_noise_texture(vvlic_ctx* c, NoiseTex& n, cudaStream_t s) {
  cudaMemcpy3DParms cp;
  std::memset(&cp, 0, sizeof cp);
  cp.srcPtr = make_cudaPitchedPtr(n.d_texels, (size_t)n.m[0] * n.ch, n.m[0], n.m[1]);
  cp.dstArray = n.array;
  cp.extent = make_cudaExtent(n.m[0], n.m[1], n.m[2]);
  cp.kind = cudaMemcpyDeviceToDevice;
  cudaError_t e = cudaMemcpy3DAsync(&cp, s);
  if (e != cudaSuccess) return cuda_fail(c, e, "noise texture copy");
  return VVLIC_OK;
}

vvlic_status ensure_noise_texture(vvlic_ctx* c, NoiseTex& n, cudaStream_t s) {
  if (n.tex) return VVLIC_OK;
  cudaChannelFormatDesc desc =
      n.ch == 4 ? cudaCreateChannelDesc<uchar4>() : cudaCreateChannelDesc<unsigned char>();
  cudaExtent ext = make_cudaExtent(n.m[0], n.m[1], n.m[2]);
  cudaError_t e = cudaMalloc3DArray(&n.array, &desc, ext);
  if (e != cudaSuccess) return cuda_fail(c, e, "noise texture allocation");
  vvlic_status st = copy_noise_texture(c, n, s);
  if (st) return st;
  cudaResourceDesc rd;
  std::memset(&rd, 0, sizeof rd);
  rd.resType = cudaResourceTypeArray;
  rd.res.array.array = n.array;
  cudaTextureDesc td;
  std::memset(&td, 0, sizeof td);
  td.addressMode[0] = td.addressMode[1] = td.addressMode[2] = cudaAddressModeWrap;
  td.filterMode = cudaFilterModeLinear;
  td.readMode = cudaReadModeNormalizedFloat;
  td.normalizedCoords = 1;
  e = cudaCreateTextureObject(&n.tex, &rd, &td, nullptr);
  if (e != cudaSuccess) return cuda_fail(c, e, "noise texture object");
  return VVLIC_OK;
}

}  // namespace

namespace vvlic {

vvlic_status encode_volume(vvlic_ctx* c, Volume& v, const void* d_xyz, int dtype, cudaStream_t s) {
  const FieldSurfaces arr = surfaces(v);
  cudaError_t e = launch_encode_field(d_xyz, dtype, v.n, v.storage, v.d_texels, c->d_scratch_word,
                                      v.array_bytes ? &arr : nullptr, s);
  if (e != cudaSuccess) return cuda_fail(c, e, "field encoding");
  if (v.d_cells) {
    e = launch_build_field_cells(v.d_texels, v.n, v.storage, v.d_cells, s);
    if (e != cudaSuccess) return cuda_fail(c, e, "cell layout rebuild");
  }
  return VVLIC_OK;
}

vvlic_status refresh_noise_layouts(vvlic_ctx* c, NoiseTex& n, cudaStream_t s) {
  if (n.d_cells) {
    cudaError_t e = launch_build_noise_cells(n.d_texels, n.m, n.ch, n.d_cells, s);
    if (e != cudaSuccess) return cuda_fail(c, e, "noise cell rebuild");
  }
  if (n.array) return copy_noise_texture(c, n, s);
  return VVLIC_OK;
}

// Wrap form and constants of the noise cells for streamlines that start within `start` of the origin.
// They move at most h_eff per step along an axis (encoded directions lie in [-1, 1], magnitudes in
// [0, 1]).
static void set_noise_wrap(double start, RenderArgs& a) {
  a.noise_wrap = choose_noise_wrap(start, std::max(a.lb, a.lf) * std::fabs((double)a.h_eff), a.nscale, a.nscale_grad, a.m);
  for (int i = 0; i < 3; ++i) noise_wrap_constants(a.m[i], &a.nclamp[i], &a.nwrap_mul[i], &a.nwrap_off[i]);
}

// Samples of the ray through pixel position (u, v) if nothing ends it: ray_setup and outside_box in double; 0 if it
// misses.
static double ray_samples(const RenderArgs& a, double u, double v) {
  double o[3], d[3], tn = -INFINITY, tf = INFINITY, len = 0.0;
  for (int i = 0; i < 3; ++i) {
    o[i] = a.o0[i] + u * a.o1[i] + v * a.o2[i];
    d[i] = a.d0[i] + u * a.d1[i] + v * a.d2[i];
    len += d[i] * d[i];
    const double t0 = -o[i] / d[i], t1 = (a.ext[i] - o[i]) / d[i];  // d = 0: a slab's infinities, or NaN, which drop out
    tn = std::fmax(tn, std::fmin(t0, t1));
    tf = std::fmin(tf, std::fmax(t0, t1));
  }
  if (a.clamp0) tn = std::fmax(tn, 0.0);
  if (!(tn < tf)) return 0.0;
  double run = INFINITY;
  for (int i = 0; i < 3; ++i) {
    const double p = (o[i] + tn * d[i]) * a.scale_vol[i], step = d[i] / std::sqrt(len) * a.scale_vol[i] * a.step_size;
    if (step != 0.0) run = std::fmin(run, ((step > 0.0 ? a.tex_max[i] : 0.0) - p) / step);
  }
  return run < 1e9 ? std::fmax(run, 1.0) : 1e9;
}

// What the work split goes by (launch_one, lane_per_ray, launch_tech_one, batches); results do not depend on it.
//   end_share: the share of all pairs of a TF alpha and an opacity that exceed the threshold (shade's alpha
//     correction undone on it).  Rays may well end early from a 64th on; a lower bar takes in random and default
//     tables whose extremes alone exceed it, whose rays go on.  At 1 every sample ends its ray.
//   along_rows: rows of pixels run (within eight degrees) along x.
//   mean_samples: the box's volume over its projection along the view axis, in samples; where the lit shaders'
//     scale makes rays march through another box than they enter (thin volumes), the mean of nine rays.
static float end_share(const vvlic_ctx* c, double thr, double alpha_corr) {
  const double bar = thr >= 1.0 ? 2.0 : (thr < 0.0 ? -1.0 : 1.0 - std::pow(1.0 - thr, 1.0 / alpha_corr));
  constexpr int n = VVLIC_TF_ENTRIES;
  const float *alpha = c->tf_sorted, *opacity = c->tf_sorted + n;  // ascending
  int pairs = 0;
  for (int i = 0, j = n; i < n; ++i) {  // as alpha grows, ever lower opacities reach the bar
    while (j > 0 && (double)alpha[i] * opacity[j - 1] > bar) --j;
    pairs += n - j;
  }
  return (float)pairs / (n * n);
}

static void set_ray_length(vvlic_ctx* c, RenderArgs& a) {
  if (c->share_thr != a.alpha_thr || c->share_corr != a.alpha_corr) {  // NaN after set_tf
    c->share = end_share(c, a.alpha_thr, a.alpha_corr);
    c->share_thr = a.alpha_thr;
    c->share_corr = a.alpha_corr;
  }
  a.end_share = c->share;
  const float* row = a.clamp0 ? a.d1 : a.o1;
  a.along_rows = row[0] * row[0] > 0.98f * (row[0] * row[0] + row[1] * row[1] + row[2] * row[2]);
  double v[3], e[3], len = 0.0, area = 0.0;
  for (int i = 0; i < 3; ++i) {
    v[i] = a.d0[i] + 0.5 * a.W * a.d1[i] + 0.5 * a.H * a.d2[i];
    e[i] = (double)a.tex_max[i] / a.scale_vol[i];  // what the ray marches through, in object space
    len += v[i] * v[i];
  }
  for (int i = 0; i < 3; ++i) area += std::fabs(v[i]) * e[(i + 1) % 3] * e[(i + 2) % 3];
  const double mean = e[0] * e[1] * e[2] * std::sqrt(len) / area / a.step_size;
  a.mean_samples = mean > 0.0 && mean < 1e9 ? (float)mean : 1e9f;
  bool same = true;
  for (int i = 0; i < 3; ++i) same = same && std::fabs(e[i] - a.ext[i]) < 1e-3 * a.ext[i];
  if (same) return;
  double sum = 0.0;
  int hits = 0;
  for (int k = 0; k < 9; ++k) {
    const double s = ray_samples(a, a.W * (k % 3 + 0.5) / 3.0, a.H * (k / 3 + 0.5) / 3.0);
    sum += s;
    hits += s > 0.0;
  }
  a.mean_samples = hits ? (float)(sum / hits) : 1e9f;
}

// Fill the kernel argument block for one volume and image size.
vvlic_status build_render_args(vvlic_ctx* c, Volume& v, int W, int H, cudaStream_t s, RenderArgs& a) {
  return build_render_args_ex(c, v, W, H, s, c->params, c->view, nullptr, a);
}

vvlic_status build_render_args_ex(vvlic_ctx* c, Volume& v, int W, int H, cudaStream_t s, const vvlic_params& p,
                                  const vvlic_view& view, const JobFilter* filter, RenderArgs& a) {
  std::memset(&a, 0, sizeof a);
  if (!c->noise.d_texels) return fail(c, VVLIC_ERR_NOT_READY, "render: no noise uploaded");
  if (p.illum == VVLIC_ILLUM_GRADIENT && c->noise.ch != 4)
    return fail(c, VVLIC_ERR_NOT_READY, "render: gradient lighting needs noise uploaded with gradients");
  if (p.scalar_gate && !c->d_scalar) return fail(c, VVLIC_ERR_NOT_READY, "render: scalar gate on, no scalar volume");
  int lb = p.low_res ? 15 : p.steps_backward, lf = p.low_res ? 15 : p.steps_forward;
  float inv_area = 0.5f;
  if (filter) {
    derive_taps_from_table(filter->table, filter->width, filter->clamp, filter->is_box, lb, lf, a.taps, &inv_area);
  } else if (derive_taps(c, lb, lf, a.taps, &inv_area)) {
    return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "render: explicit taps were set for L_b=%d L_f=%d, params have %d/%d",
                c->taps_lb, c->taps_lf, lb, lf);
  }
  vvlic_status st;
  a.n[0] = v.n[0];
  a.n[1] = v.n[1];
  a.n[2] = v.n[2];
  switch (p.sampler) {
    case VVLIC_SAMPLER_GATHER:
    case VVLIC_SAMPLER_BRICK:  // bricks are staged from the texel arrays; fetches outside them gather
      a.field = v.d_texels;
      a.noise = c->noise.d_texels;
      break;
    case VVLIC_SAMPLER_CELL:
      if ((st = ensure_cells(c, v, s))) return st;
      if ((st = ensure_noise_cells(c, c->noise, s))) return st;
      a.field = v.d_cells;
      a.noise = c->noise.d_cells;
      break;
    case VVLIC_SAMPLER_TEXTURE:
      if ((st = ensure_texture(c, v, s))) return st;
      if ((st = ensure_noise_texture(c, c->noise, s))) return st;
      a.tex = v.tex[0];
      a.tex_z = v.tex[1];
      a.tex_w = v.tex[2];
      a.noise_tex = c->noise.tex;
      break;
    default:  // HYBRID
      if ((st = ensure_texture(c, v, s))) return st;
      if ((st = ensure_noise_cells(c, c->noise, s))) return st;
      a.tex = v.tex[0];
      a.tex_z = v.tex[1];
      a.tex_w = v.tex[2];
      a.noise = c->noise.d_cells;
      break;
  }

  const bool cells = p.sampler == VVLIC_SAMPLER_CELL || p.sampler == VVLIC_SAMPLER_HYBRID;
  for (int i = 0; i < 3; ++i) {
    a.m[i] = cells ? noise_cell_extent(c->noise.m[i]) : c->noise.m[i];
    a.sn[i] = c->sn[i];
  }
  a.noise_ch = c->noise.ch;
  a.scalar = c->d_scalar;
  a.tf = c->d_tf;
  a.W = W;
  a.H = H;
  double rc[21];
  derive_rays(view, v.geom, W, H, rc);
  for (int i = 0; i < 3; ++i) {
    a.o0[i] = (float)rc[i];
    a.o1[i] = (float)rc[3 + i];
    a.o2[i] = (float)rc[6 + i];
    a.d0[i] = (float)rc[9 + i];
    a.d1[i] = (float)rc[12 + i];
    a.d2[i] = (float)rc[15 + i];
  }
  a.clamp0 = rc[18] != 0.0;
  // scaleVol / scaleVolInv as the shader receives them (renderer.cpp:939-944)
  const bool bug = (p.quirks & VVLIC_QUIRK_UNIFORM_SCALE_BUG) && p.illum != VVLIC_ILLUM_NONE;
  for (int i = 0; i < 3; ++i) {
    a.ext[i] = v.geom.extent[i];
    a.tex_max[i] = v.geom.tex_max[i];
    a.scale_vol[i] = bug ? v.geom.scale_inv[i] : v.geom.scale[i];
    a.scale_vol_inv[i] = bug ? 0.0f : v.geom.scale_inv[i];
  }
  const float h = p.low_res ? 1.0f / 64.0f : p.step_size_lic;
  a.step_size = p.low_res ? 2.0f * p.step_size_vol : p.step_size_vol;
  a.freq_scale = p.low_res ? 0.7f * p.freq_scale : p.freq_scale;
  const bool nofreq = (p.quirks & VVLIC_QUIRK_GRAD_NOISE_NO_FREQ) != 0;
  for (int i = 0; i < 3; ++i) {
    a.nscale[i] = (float)((double)a.freq_scale * c->noise.m[i]);
    a.nscale_grad[i] = nofreq ? (float)c->noise.m[i] : a.nscale[i];
  }
  a.alpha_corr = p.low_res ? 2.0f * p.step_size_vol * 128.0f : p.step_size_vol * 128.0f;
  a.h_eff = h * p.eye_dist_factor;
  a.intensity_scale = inv_area / (float)(lf + lb) * p.gradient_scale;  // licKernel.b * gradient.r
  a.illum_scale = p.illum_scale;
  a.alpha_thr = p.alpha_threshold;
  set_ray_length(c, a);
  a.gate_lo = p.gate_lo;
  a.gate_hi = p.gate_hi;
  a.num_iter = p.num_iterations;
  a.lb = lb;
  a.lf = lf;
  double origin = 0.0, dir = 0.0;
  for (int i = 0; i < 3; ++i) {
    origin = larger(origin, std::fabs((double)a.o0[i]) + W * std::fabs((double)a.o1[i]) + H * std::fabs((double)a.o2[i]));
    if (!a.clamp0) dir = larger(dir, std::fabs((double)a.d0[i]));
  }
  set_noise_wrap(ray_start_bound(a.ext, a.scale_vol, a.tex_max, origin, dir), a);
  a.illum = p.illum;
  a.tf_index = p.tf_index;
  a.sof = p.speed_of_flow;
  a.gate = p.scalar_gate;
  a.quirks = (int)p.quirks;
  a.spec_exp = p.spec_exp;
  for (int i = 0; i < 3; ++i) {
    a.light_pos[i] = p.light_pos[i];
    a.light_diff[i] = p.light_diffuse[i];
    a.light_spec[i] = p.light_specular[i];
    a.light_amb[i] = p.light_ambient[i];
  }
  if (p.illum == VVLIC_ILLUM_ZOECKLER || p.illum == VVLIC_ILLUM_MALLO) {
    if ((st = ensure_illum_luts(c)) != VVLIC_OK) return st;
    a.luts = (const uchar4*)c->d_luts;
    a.lut_w = c->lut_w;
    a.lut_h = c->lut_h;
  }
  a.counters = c->d_counters;
  return VVLIC_OK;
}

cudaError_t launch_technique(int storage, const RenderArgs& a, const TechArgs& t, int sampler, int integ, bool grad,
                             int num_sms, cudaStream_t s) {
  switch (kernel_storage(storage, sampler)) {
    case VVLIC_STORAGE_F32: return launch_technique_f32(a, t, sampler, integ, grad, num_sms, s);
    case VVLIC_STORAGE_F16: return launch_technique_f16(a, t, sampler, integ, grad, num_sms, s);
    case VVLIC_STORAGE_UNORM8: return launch_technique_u8(a, t, sampler, integ, grad, num_sms, s);
    default: return launch_technique_bf16(a, t, sampler, integ, grad, num_sms, s);
  }
}

cudaError_t launch_raycast(const RenderArgs& a, int storage, int sampler, int integ, bool grad, int num_sms,
                           cudaStream_t s) {
  switch (kernel_storage(storage, sampler)) {
    case VVLIC_STORAGE_F32: return launch_raycast_f32(a, sampler, integ, grad, num_sms, s);
    case VVLIC_STORAGE_F16: return launch_raycast_f16(a, sampler, integ, grad, num_sms, s);
    case VVLIC_STORAGE_UNORM8: return launch_raycast_u8(a, sampler, integ, grad, num_sms, s);
    default: return launch_raycast_bf16(a, sampler, integ, grad, num_sms, s);
  }
}

}  // namespace vvlic

namespace {

// Tape buffers for a recording render: per ray `stride` samples (the longest march / spacing,
// capped by the two loop bounds) and a checkpoint every kSegment samples.  A ray marches in
// texture space through [0, tex_max] by step_size * |normalize(d) * scaleVol| per sample, and
// that step is at least step_size * min(scaleVol): the bound holds whatever scaleVol the
// shader receives (with VVLIC_QUIRK_UNIFORM_SCALE_BUG it is scaleInv, and rays run past the
// object box until they leave [0, tex_max]).
vvlic_status prepare_tape(vvlic_ctx* c, int w, int h, RenderArgs& a, cudaStream_t s) {
  const double diag = std::sqrt((double)a.tex_max[0] * a.tex_max[0] + (double)a.tex_max[1] * a.tex_max[1] +
                                (double)a.tex_max[2] * a.tex_max[2]);
  const double min_sv = std::max(1e-6, (double)std::min(std::min(a.scale_vol[0], a.scale_vol[1]), a.scale_vol[2]));
  double bound = std::min(diag / (a.step_size * min_sv) + 3.0, (double)a.num_iter * (double)a.num_iter);
  if (c->params.tape_max_samples > 0) bound = std::min(bound, (double)c->params.tape_max_samples);
  const int stride = std::max(1, (int)std::ceil(bound));
  const int nck = (stride + kSegment - 1) / kSegment;
  const size_t rays = (size_t)w * h;
  // per-sample arrays in 8x4-ray tiles (tape_entry / tape_ck_entry), edge tiles padded
  const size_t slots = (size_t)((w + 7) / 8) * (size_t)((h + 3) / 4) * 32;
  const bool lit = a.illum == VVLIC_ILLUM_GRADIENT;
  const size_t b_is = slots * stride * sizeof(float2), b_ck = slots * nck * 2 * sizeof(float4),
               b_g = lit ? slots * stride * sizeof(uint2) : 0, b_n = rays * sizeof(uint32_t);
  const size_t bytes = b_ck + b_is + b_g + b_n;
  if (c->tape_cap < bytes) {
    if (c->d_tape) cudaFree(c->d_tape);
    c->d_tape = nullptr;
    c->tape_cap = 0;
    cudaError_t e = cudaMalloc(&c->d_tape, bytes);
    if (e != cudaSuccess) return cuda_fail(c, e, "adjoint tape allocation");
    c->tape_cap = bytes;
  }
  if (!c->d_tape_flag) {
    cudaError_t e = cudaMalloc(&c->d_tape_flag, sizeof(unsigned long long));
    if (e != cudaSuccess) return cuda_fail(c, e, "adjoint tape flag");
  }
  char* base = (char*)c->d_tape;
  a.tape_ck = (float4*)base;
  a.tape_is = (float2*)(base + b_ck);
  a.tape_g = lit ? (uint2*)(base + b_ck + b_is) : nullptr;
  a.tape_n = (uint32_t*)(base + b_ck + b_is + b_g);
  a.tape_overflow = c->d_tape_flag;
  a.tape_stride = stride;
  a.tape_nck = nck;
  cudaError_t e = cudaMemsetAsync(c->d_tape_flag, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return cuda_fail(c, e, "adjoint tape flag");
  return VVLIC_OK;
}

}  // namespace

extern "C" vvlic_status vvlic_render_device(vvlic_ctx* c, int32_t vol_id, float* d_out, int32_t w, int32_t h,
                                           uint32_t* d_samples, void* stream) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  auto it = c->vols.find(vol_id);
  if (it == c->vols.end()) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "render: unknown volume %d", vol_id);
  if (!d_out || w < 1 || h < 1 || w > 32768 || h > 32768)
    return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "render: bad image arguments");
  DeviceGuard g(c->device);
  cudaStream_t s = (cudaStream_t)stream;
  RenderArgs a;
  vvlic_status st = build_render_args(c, it->second, w, h, s, a);
  if (st) return st;
  a.out = d_out;
  a.samples = d_samples;
  if (c->params.sampler == VVLIC_SAMPLER_BRICK &&
      (c->params.technique != VVLIC_TECHNIQUE_RAYCAST || c->params.record_tape))
    return fail(c, VVLIC_ERR_UNSUPPORTED, "render: the BRICK sampler renders the RAYCAST technique without a tape");
  if (c->params.technique != VVLIC_TECHNIQUE_RAYCAST) {
    if (c->params.record_tape)
      return fail(c, VVLIC_ERR_UNSUPPORTED, "render: the adjoint tape is recorded by the RAYCAST technique only");
    TechArgs t;
    std::memset(&t, 0, sizeof t);
    t.technique = c->params.technique;
    const Volume& v = it->second;
    if (t.technique == VVLIC_TECHNIQUE_SLICING) {
      derive_slicing(c->view, v.geom, a.step_size, t.v, &t.depth, &t.nslices);
      for (int i = 0; i < 3; ++i) t.c[i] = v.geom.center[i];
    } else if (t.technique == VVLIC_TECHNIQUE_LICVOLUME) {
      if (!v.d_licvol || !v.licvol_valid)
        return fail(c, VVLIC_ERR_NOT_READY, "render: LICVOLUME needs vvlic_compute_lic_volume for volume %d", vol_id);
      t.licvol = v.d_licvol;
      for (int i = 0; i < 3; ++i) t.ln[i] = v.ln[i];
      a.illum = VVLIC_ILLUM_NONE;  // raycast_lic3d_fragment.glsl shades with illumLIC
    }
    cudaError_t e = cudaMemsetAsync(c->d_counters, 0, 4 * sizeof(unsigned long long), s);
    if (e == cudaSuccess) e = cudaEventRecord(c->ev0, s);
    if (e == cudaSuccess)
      e = launch_technique(v.storage, a, t, c->params.sampler, c->params.integrator,
                           c->params.illum == VVLIC_ILLUM_GRADIENT && t.technique == VVLIC_TECHNIQUE_SLICING, c->num_sms,
                           s);
    if (e == cudaSuccess) e = cudaEventRecord(c->ev1, s);
    if (e != cudaSuccess) return cuda_fail(c, e, "render launch");
    c->stats_pending = true;
    c->last_was_batch = false;
    c->tape_flag_pending = false;
    c->stats_steps_per_sample = t.technique == VVLIC_TECHNIQUE_SLICING ? (uint64_t)(a.lb + a.lf) : 0;
    return VVLIC_OK;
  }
  const bool record = c->params.record_tape != 0;
  if (record) {
    c->tape_valid = false;
    if ((st = prepare_tape(c, w, h, a, s))) return st;
  }
  const bool grad = c->params.illum == VVLIC_ILLUM_GRADIENT;
  const bool brick = c->params.sampler == VVLIC_SAMPLER_BRICK;
  BrickArgs bargs;
  if (brick && (st = prepare_brick(c, it->second, a, grad, bargs))) return st;
  cudaError_t e = cudaMemsetAsync(c->d_counters, 0, 4 * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return cuda_fail(c, e, "render");
  e = cudaEventRecord(c->ev0, s);
  if (e == cudaSuccess)
    e = brick ? launch_brick(it->second.storage, a, bargs, c->params.integrator, grad, s)
              : launch_raycast(a, it->second.storage, c->params.sampler, c->params.integrator, grad, c->num_sms, s);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev1, s);
  if (e != cudaSuccess) return cuda_fail(c, e, "render launch");
  c->stats_pending = true;
  c->last_was_batch = false;
  c->stats.sample_steps = 0;
  c->stats_steps_per_sample = (uint64_t)(a.lb + a.lf);
  c->tape_flag_pending = record;
  if (record) {
    c->tape_valid = true;
    c->tape_vol = vol_id;
    c->tape_w = w;
    c->tape_h = h;
    c->tape_storage = it->second.storage;
    c->tape_sampler = c->params.sampler;
    c->tape_integ = c->params.integrator;
    c->tape_illum = c->params.illum;
    c->tape_args = a;
  }
  return VVLIC_OK;
}

namespace vvlic_adjoint_out {

__global__ void fixed_to_float_kernel(const long long* acc, int n_tf, int n_op, int n_taps, float* tf, float* op,
                                      float* taps, const unsigned long long* overflow) {
  const float nan = __int_as_float(0x7fc00000);
  const bool bad = *overflow != 0;
  const double k = 1.0 / 1073741824.0;  // 2^-30
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_tf + n_op + n_taps; i += gridDim.x * blockDim.x) {
    const float v = bad ? nan : (float)((double)acc[i] * k);
    if (i < n_tf) {
      if (tf) tf[i] = v;
    } else if (i < n_tf + n_op) {
      if (op) op[i - n_tf] = v;
    } else if (taps) {
      taps[i - n_tf - n_op] = v;
    }
  }
}

}  // namespace vvlic_adjoint_out

extern "C" vvlic_status vvlic_render_adjoint(vvlic_ctx* c, int32_t vol_id, const float* d_dl_drgba, int32_t w,
                                            int32_t h, float* d_dl_dtf, float* d_dl_dopacity, float* d_dl_dtaps,
                                            void* stream) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  if (!d_dl_drgba) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "render_adjoint: null cotangent");
  if (!c->tape_valid || c->tape_vol != vol_id || c->tape_w != w || c->tape_h != h)
    return fail(c, VVLIC_ERR_NOT_READY,
                "render_adjoint: the last render of this context did not record a tape for volume %d at %dx%d "
                "(set params.record_tape)", vol_id, w, h);
  if (c->vols.find(vol_id) == c->vols.end())
    return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "render_adjoint: unknown volume %d", vol_id);
  DeviceGuard g(c->device);
  cudaStream_t s = (cudaStream_t)stream;
  const int acc_size = 5 * VVLIC_TF_ENTRIES + kMaxTaps;
  cudaError_t e = cudaSuccess;
  if (!c->d_acc) {
    e = cudaMalloc(&c->d_acc, (acc_size + 1) * sizeof(long long));  // the accumulators and the queue counter
    if (e != cudaSuccess) return cuda_fail(c, e, "adjoint accumulators");
  }
  e = cudaMemsetAsync(c->d_acc, 0, (acc_size + 1) * sizeof(long long), s);
  if (e != cudaSuccess) return cuda_fail(c, e, "adjoint");
  const RenderArgs& a = c->tape_args;
  unsigned* next = reinterpret_cast<unsigned*>(c->d_acc + acc_size);
  const int sms = c->num_sms;
  e = cudaEventRecord(c->ev0, s);
  const float4* gi = (const float4*)d_dl_drgba;
  if (e == cudaSuccess) {
    const bool lit = c->tape_illum == VVLIC_ILLUM_GRADIENT;
    switch (kernel_storage(c->tape_storage, c->tape_sampler)) {
      case VVLIC_STORAGE_F32: e = launch_adjoint_f32(a, c->tape_sampler, c->tape_integ, lit, gi, c->d_acc, next, sms, s); break;
      case VVLIC_STORAGE_F16: e = launch_adjoint_f16(a, c->tape_sampler, c->tape_integ, lit, gi, c->d_acc, next, sms, s); break;
      case VVLIC_STORAGE_UNORM8:
        e = launch_adjoint_u8(a, c->tape_sampler, c->tape_integ, lit, gi, c->d_acc, next, sms, s);
        break;
      default: e = launch_adjoint_bf16(a, c->tape_sampler, c->tape_integ, lit, gi, c->d_acc, next, sms, s); break;
    }
  }
  if (e == cudaSuccess) e = cudaEventRecord(c->ev1, s);
  if (e == cudaSuccess) {
    const int n_taps = a.lb + a.lf + 1;
    vvlic_adjoint_out::fixed_to_float_kernel<<<8, 256, 0, s>>>(c->d_acc, 4 * VVLIC_TF_ENTRIES, VVLIC_TF_ENTRIES, n_taps, d_dl_dtf,
                                            d_dl_dopacity, d_dl_dtaps, c->d_tape_flag);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "render_adjoint launch");
  c->stats_pending = true;
  c->tape_flag_pending = true;
  return VVLIC_OK;
}

extern "C" vvlic_status vvlic_render(vvlic_ctx* c, int32_t vol_id, float* out, int32_t w, int32_t h) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  if (!out || w < 1 || h < 1 || w > 32768 || h > 32768)
    return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "render: bad image arguments");
  DeviceGuard g(c->device);
  const size_t bytes = (size_t)w * h * 4 * sizeof(float);
  if (c->image_cap < bytes) {
    if (c->d_image) cudaFree(c->d_image);
    c->d_image = nullptr;
    c->image_cap = 0;
    cudaError_t e = cudaMalloc(&c->d_image, bytes);
    if (e != cudaSuccess) return cuda_fail(c, e, "image allocation");
    c->image_cap = bytes;
  }
  vvlic_status st = vvlic_render_device(c, vol_id, (float*)c->d_image, w, h, nullptr, c->stream);
  if (st) return st;
  cudaError_t e = cudaMemcpyAsync(out, c->d_image, bytes, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "render");
  return VVLIC_OK;
}

extern "C" vvlic_status vvlic_render_to_host_async(vvlic_ctx* c, int32_t vol_id, float* out, int32_t w, int32_t h,
                                                  void* stream) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  if (!out || w < 1 || h < 1 || w > 32768 || h > 32768)
    return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "render_to_host_async: bad image arguments");
  DeviceGuard g(c->device);
  const size_t bytes = (size_t)w * h * 4 * sizeof(float);
  if (c->image_cap < bytes) {
    cudaError_t e = cudaDeviceSynchronize();  // a download in flight may still read the image
    if (e != cudaSuccess) return cuda_fail(c, e, "render_to_host_async");
    if (c->d_image) cudaFree(c->d_image);
    c->d_image = nullptr;
    c->image_cap = 0;
    e = cudaMalloc(&c->d_image, bytes);
    if (e != cudaSuccess) return cuda_fail(c, e, "image allocation");
    c->image_cap = bytes;
  }
  vvlic_status st = vvlic_render_device(c, vol_id, (float*)c->d_image, w, h, nullptr, stream);
  if (st) return st;
  cudaError_t e = cudaMemcpyAsync(out, c->d_image, bytes, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "render_to_host_async");
  return VVLIC_OK;
}

extern "C" vvlic_status vvlic_get_stats(vvlic_ctx* c, vvlic_stats* out) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  if (!out) return VVLIC_ERR_INVALID_ARGUMENT;
  if (c->stats_pending) {
    DeviceGuard g(c->device);
    cudaError_t e = cudaEventSynchronize(c->ev1);
    unsigned long long h[4];
    if (e == cudaSuccess) e = cudaMemcpy(h, c->d_counters, sizeof h, cudaMemcpyDeviceToHost);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    if (e != cudaSuccess) return cuda_fail(c, e, "get_stats");
    c->stats.samples = h[0];
    c->stats.rays = h[1];
    // a batch mixes LIC lengths and counts its sample-steps on the device
    c->stats.sample_steps = c->last_was_batch ? h[2] : h[0] * c->stats_steps_per_sample;
    c->stats.kernel_ms = ms;
    c->stats.check_flags = (uint32_t)h[3];
    if (c->tape_flag_pending && c->d_tape_flag) {
      // rays of the recording render that outgrew their tape (store_pixel counts them)
      unsigned long long over = 0;
      e = cudaMemcpy(&over, c->d_tape_flag, sizeof over, cudaMemcpyDeviceToHost);
      if (e != cudaSuccess) return cuda_fail(c, e, "get_stats");
      if (over) c->stats.check_flags |= VVLIC_CHECK_TAPE_OVERFLOW;
    }
    c->stats_pending = false;
  }
  *out = c->stats;
  return VVLIC_OK;
}

extern "C" vvlic_status vvlic_compute_lic_volume(vvlic_ctx* c, int32_t vol_id, int32_t nx, int32_t ny, int32_t nz) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  auto it = c->vols.find(vol_id);
  if (it == c->vols.end()) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "compute_lic_volume: unknown volume %d", vol_id);
  if (nx < 1 || ny < 1 || nz < 1 || nx > 2048 || ny > 2048 || nz > 2048)
    return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "compute_lic_volume: dims");
  if (c->params.sampler == VVLIC_SAMPLER_BRICK)
    return fail(c, VVLIC_ERR_UNSUPPORTED, "compute_lic_volume: the BRICK sampler renders the RAYCAST technique only");
  DeviceGuard g(c->device);
  Volume& v = it->second;
  cudaStream_t s = c->stream;
  RenderArgs a;
  vvlic_status st = build_render_args(c, v, 1, 1, s, a);
  if (st) return st;
  const size_t count = (size_t)nx * ny * nz;
  if (v.d_licvol && (size_t)v.ln[0] * v.ln[1] * v.ln[2] != count) {
    cudaStreamSynchronize(s);
    cudaFree(v.d_licvol);
    v.d_licvol = nullptr;
  }
  if (!v.d_licvol) {
    cudaError_t e = cudaMalloc(&v.d_licvol, count * sizeof(float));
    if (e != cudaSuccess) return cuda_fail(c, e, "LIC volume allocation");
  }
  v.ln[0] = nx;
  v.ln[1] = ny;
  v.ln[2] = nz;
  TechArgs t;
  std::memset(&t, 0, sizeof t);
  t.technique = VVLIC_TECHNIQUE_LICVOLUME;
  t.licvol_out = v.d_licvol;
  t.ln[0] = nx;
  t.ln[1] = ny;
  t.ln[2] = nz;
  // lic3d_volume_fragment.glsl composes inc_lic without inc_illum: the uniform scaleVol is the
  // volume's scale whatever the shading variant
  for (int i = 0; i < 3; ++i) a.scale_vol[i] = v.geom.scale[i];
  set_noise_wrap(voxel_start_bound(a.scale_vol), a);  // streamlines start at voxels, not on rays
  cudaError_t e = cudaMemsetAsync(c->d_counters, 0, 4 * sizeof(unsigned long long), s);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev0, s);
  if (e == cudaSuccess) e = launch_technique(v.storage, a, t, c->params.sampler, c->params.integrator, false, c->num_sms, s);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev1, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(c, e, "compute_lic_volume");
  v.licvol_valid = true;
  // the precompute's statistics: one LIC sample per voxel, L_b + L_f streamline steps each
  unsigned long long h[4];
  float ms = 0.f;
  e = cudaMemcpy(h, c->d_counters, sizeof h, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  if (e != cudaSuccess) return cuda_fail(c, e, "compute_lic_volume statistics");
  c->stats.samples = count;
  c->stats.sample_steps = count * (uint64_t)(a.lb + a.lf);
  c->stats.rays = 0;
  c->stats.kernel_ms = ms;
  c->stats.check_flags = (uint32_t)h[3];
  c->stats_pending = false;
  c->last_was_batch = false;
  c->tape_flag_pending = false;
  return VVLIC_OK;
}

extern "C" vvlic_status vvlic_download_lic_volume(vvlic_ctx* c, int32_t vol_id, float* out, uint64_t capacity) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  auto it = c->vols.find(vol_id);
  if (it == c->vols.end() || !it->second.d_licvol || !it->second.licvol_valid)
    return fail(c, VVLIC_ERR_NOT_READY, "download_lic_volume: no LIC volume for volume %d", vol_id);
  const size_t bytes = (size_t)it->second.ln[0] * it->second.ln[1] * it->second.ln[2] * sizeof(float);
  if (!out || capacity < bytes) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "download_lic_volume: need %zu bytes", bytes);
  DeviceGuard g(c->device);
  cudaError_t e = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess) e = cudaMemcpy(out, it->second.d_licvol, bytes, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(c, e, "download_lic_volume");
  return VVLIC_OK;
}

extern "C" vvlic_status vvlic_synchronize(vvlic_ctx* c, void* stream, int32_t timeout_ms) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  if (timeout_ms < 0) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "synchronize: negative timeout");
  DeviceGuard g(c->device);
  const auto deadline = std::chrono::steady_clock::now() + std::chrono::microseconds((int64_t)timeout_ms * 1000);
  cudaStream_t streams[2] = {(cudaStream_t)stream, c->stream};
  for (cudaStream_t st : streams) {
    for (;;) {
      const cudaError_t e = cudaStreamQuery(st);
      if (e == cudaSuccess) break;
      if (e != cudaErrorNotReady) return cuda_fail(c, e, "synchronize");
      if (std::chrono::steady_clock::now() >= deadline)
        return fail(c, VVLIC_ERR_TIMEOUT, "synchronize: work still running after %d ms", timeout_ms);
      std::this_thread::sleep_for(std::chrono::microseconds(50));
    }
  }
  return VVLIC_OK;
}
