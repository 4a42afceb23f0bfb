// The reference's other render techniques over the same field, noise and LIC machinery:
//   * SLICING (Renderer::sliceVolume renderer.cpp:1123-1267, ViewSlicing slicing.cpp:42-263,
//     lic3d_slicing_fragment.glsl): samples where each pixel's ray crosses the view-aligned
//     planes d_i = -D/2 + (i+1/2) D/N through the volume centre, front to back; TF on the
//     magnitude, LIC only where tf.a > 0.05, no more blending once dest.a >= 0.95.
//   * VOLUME (Renderer::renderVolume renderer.cpp:1066-1090, vectorfield_fragment.glsl:39-101):
//     direct volume rendering of the encoded directions, src = (field.rgb, TF(field.a).a).
//   * LICVOLUME (Renderer::renderLICVolume renderer.cpp:1311-1374 + lic3d_volume_fragment.glsl,
//     then raycast_lic3d_fragment.glsl): a precomputed volume of LIC intensities (one per voxel
//     centre), ray-cast with illumLIC; REPEAT-wrapped like the reference's VolumeBuffer.
// VOLUME and LICVOLUME stop on the accumulated dest.a > 0.95 as their shaders do.
#pragma once

#include "render_fwd.cuh"

namespace vvlic {

// texture3D(licVolumeSampler, s).r: LINEAR + REPEAT (VolumeBuffer.cpp:43-57), in FP32.
__device__ __forceinline__ float sample_licvol(const TechArgs& t, float3 s) {
  int x0, x1, y0, y1, z0, z1;
  float ax, ay, az;
  repeat_axis_fast(s.x, t.ln[0], x0, x1, ax);
  repeat_axis_fast(s.y, t.ln[1], y0, y1, ay);
  repeat_axis_fast(s.z, t.ln[2], z0, z1, az);
  // up to 2048^3 entries: row offsets in 64 bits
  const size_t nx = (size_t)t.ln[0], nxy = nx * (size_t)t.ln[1];
  const float* v = t.licvol;
  const float* r00 = v + z0 * nxy + y0 * nx;
  const float* r10 = v + z0 * nxy + y1 * nx;
  const float* r01 = v + z1 * nxy + y0 * nx;
  const float* r11 = v + z1 * nxy + y1 * nx;
  const float c00 = lerpf(__ldg(r00 + x0), __ldg(r00 + x1), ax);
  const float c10 = lerpf(__ldg(r10 + x0), __ldg(r10 + x1), ax);
  const float c01 = lerpf(__ldg(r01 + x0), __ldg(r01 + x1), ax);
  const float c11 = lerpf(__ldg(r11 + x0), __ldg(r11 + x1), ax);
  return lerpf(lerpf(c00, c10, ay), lerpf(c01, c11, ay), az);
}

// SLICING by a warp on 32 / S rays, S lanes to a ray.  The lanes test S planes of their ray at a time
// (inside the slice polygon, TF alpha above 0.05) and queue those that pass; once every ray has S
// or no planes left, each lane computes one queued plane's LIC and the ray's lanes composite them
// in order.  So the streamline work, nearly all of the cost, runs in full groups however few planes
// pass; a lane per pixel idles wherever its own plane does not (18.5 of 32 lanes active).  Planes, order,
// arithmetic and counts are those of one lane walking the planes; the ones after dest.a reaches 0.95
// are dropped.  launch_tech_one has the rule and the times.
template <int ST, int FL, int NL, int INTEG, bool GRAD, int S>
__global__ void __launch_bounds__(cast_threads<INTEG>(), min_blocks<INTEG>() * 128 / cast_threads<INTEG>())
    slicing_kernel(const __grid_constant__ RenderArgs a, const __grid_constant__ TechArgs t) {
  constexpr int R = 32 / S;
  __shared__ __align__(16) float s_tf[5 * VVLIC_TF_ENTRIES];
  __shared__ int s_queue[cast_threads<INTEG>() / 32][R][2 * S];
  load_tf(a, s_tf);
  const CtaShape cta = cta_shape(blockDim.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = lane / R, r = lane % R;
  using T = GroupTile<S>;
  const int px = ((int)blockIdx.x * cta.wx + warp % cta.wx) * T::w + r % T::w;
  const int py = ((int)blockIdx.y * cta.wy + warp / cta.wx) * T::h + r / T::w;
  const unsigned mine = ray_lanes(S) << r;
  int* queue = s_queue[warp][r];
  const bool ray = px < a.W && py < a.H;
  float o[3] = {0.f, 0.f, 0.f}, d[3] = {0.f, 0.f, 0.f}, tn = 0.0f, tf = 0.0f;
  const bool hit = ray && ray_interval(a, px, py, o, d, tn, tf);
  const float3 O = f3(o[0], o[1], o[2]), D = f3(d[0], d[1], d[2]);
  const float3 V = f3(t.v[0], t.v[1], t.v[2]), C = f3(t.c[0], t.c[1], t.c[2]);
  const float vd = dot3(V, D);
  const float voc = dot3(V, sub3(O, C));
  const float3 sv = f3(a.scale_vol[0], a.scale_vol[1], a.scale_vol[2]);
  const float3 dir = mul3(norm3(D), sv);
  const float step = t.depth / (float)t.nslices;
  const auto plane = [&](int i) {  // ray parameter of plane i
    const float di = -0.5f * t.depth + ((float)i + 0.5f) * step;
    return (di - voc) / vd;
  };
  float4 dest = make_float4(0.f, 0.f, 0.f, 0.f);
  uint32_t samples = 0;
  bool open = hit && vd != 0.0f;  // vd == 0: the ray is parallel to the planes
  int next = 0, queued = 0;
  for (;;) {
    while (__any_sync(0xffffffffu, open && queued < S && next < t.nslices)) {
      const bool scan = open && queued < S && next < t.nslices;
      const int i = next + k;
      bool pass = false;
      if (scan && i < t.nslices) {
        const float ti = plane(i);
        if (ti >= tn && ti <= tf)  // inside the slice polygon (plane inside the box)
          pass = tf_rgba(s_tf, Field<ST, FL>::sample(a, mul3(add3(O, scl3(D, ti)), sv)).w).w > 0.05f;
      }
      const unsigned passed = __ballot_sync(0xffffffffu, pass) & mine;
      if (pass) queue[queued + __popc(passed & ((1u << lane) - 1u))] = i;
      queued += __popc(passed);
      if (scan) next += S;
    }
    __syncwarp();
    if (!__any_sync(0xffffffffu, open && queued > 0)) break;
    const int n = open ? min(queued, S) : 0;
    float4 src = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < n) {
      const float3 pos = mul3(add3(O, scl3(D, plane(queue[k]))), sv);
      const float4 f = Field<ST, FL>::sample(a, pos);
      const float4 tfv = tf_rgba(s_tf, f.w);
      float4 il = compute_lic<ST, FL, NL, INTEG, GRAD>(a, pos, f);
      il.w *= a.intensity_scale;
      src = shade<GRAD>(a, s_tf, il, tfv, pos, dir, f);
    }
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const float4 s = shfl4(src, j * R + r);
      if (j < n && open) {
        if (dest.w >= 0.95f) {  // lic3d_slicing_fragment.glsl:14 (no later slice changes dest)
          open = false;
        } else {
          dest = blend(dest, s);
          ++samples;
        }
      }
    }
    queued -= n;
    const int rest = k < queued ? queue[S + k] : 0;  // at most S - 1 remain behind a full group
    __syncwarp();
    if (k < queued) queue[k] = rest;
    __syncwarp();
  }
  const bool store = ray && lane < R;
  if (store) store_pixel(a, px, py, dest, samples);
  flush_counters(a, store ? samples : 0u, store && hit ? 1u : 0u);
}

// SLICING by one lane per pixel: a warp stays on one plane, whose neighbouring pixels read neighbouring texels.
template <int ST, int FL, int NL, int INTEG, bool GRAD>
__device__ __forceinline__ float4 slice_pixel(const RenderArgs& a, const TechArgs& t, const float* s_tf, int px,
                                              int py, uint32_t& samples, uint32_t& hit) {
  float4 dest = make_float4(0.f, 0.f, 0.f, 0.f);
  samples = 0;
  hit = 0;
  float o[3], d[3], tn, tf;
  if (!ray_interval(a, px, py, o, d, tn, tf)) return dest;
  hit = 1;
  const float3 O = f3(o[0], o[1], o[2]), D = f3(d[0], d[1], d[2]);
  const float3 V = f3(t.v[0], t.v[1], t.v[2]), C = f3(t.c[0], t.c[1], t.c[2]);
  const float vd = dot3(V, D);
  if (vd == 0.0f) return dest;  // ray parallel to the planes
  const float voc = dot3(V, sub3(O, C));
  const float3 sv = f3(a.scale_vol[0], a.scale_vol[1], a.scale_vol[2]);
  const float3 dir = mul3(norm3(D), sv);
  const float step = t.depth / (float)t.nslices;
  for (int i = 0; i < t.nslices; ++i) {
    if (dest.w >= 0.95f) break;  // lic3d_slicing_fragment.glsl:14 (no later slice changes dest)
    const float di = -0.5f * t.depth + ((float)i + 0.5f) * step;
    const float ti = (di - voc) / vd;
    if (!(ti >= tn && ti <= tf)) continue;  // outside the slice polygon (plane inside the box)
    const float3 pos = mul3(add3(O, scl3(D, ti)), sv);
    const float4 f = Field<ST, FL>::sample(a, pos);
    const float4 tfv = tf_rgba(s_tf, f.w);
    if (!(tfv.w > 0.05f)) continue;
    float4 il = compute_lic<ST, FL, NL, INTEG, GRAD>(a, pos, f);
    ++samples;
    il.w *= a.intensity_scale;
    dest = blend(dest, shade<GRAD>(a, s_tf, il, tfv, pos, dir, f));
  }
  return dest;
}

template <int ST, int FL, int NL, int INTEG, bool GRAD>
__global__ void __launch_bounds__(kThreads, VVLIC_MIN_BLOCKS)
    slicing_pixel_kernel(const __grid_constant__ RenderArgs a, const __grid_constant__ TechArgs t) {
  __shared__ __align__(16) float s_tf[5 * VVLIC_TF_ENTRIES];
  load_tf(a, s_tf);
  const int px = blockIdx.x * kTileW + (threadIdx.x % kTileW);
  const int py = blockIdx.y * kTileH + (threadIdx.x / kTileW);
  uint32_t samples = 0, hit = 0;
  if (px < a.W && py < a.H)
    store_pixel(a, px, py, slice_pixel<ST, FL, NL, INTEG, GRAD>(a, t, s_tf, px, py, samples, hit), samples);
  flush_counters(a, samples, hit);
}

// VOLUME / LICVOLUME for one pixel.  LICVOLUME keeps four (AHEAD) samples' fetches in flight (a texture fetch and
// eight loads each; those past the sample that ends the ray are dropped): 1024^2 frame of a 256^3 LIC
// volume 357 -> 190 us; two where rays are short or may end at once (launch_tech_layout).  A VOLUME sample is one fetch, and one at a time is as fast (1600x1200 frame of
// 512^3 59 us with 1, 2, 4 or 8 in flight; 200x150 of 64^3 with its field update 24 us against 28).
template <int ST, int FL, bool LICVOL, int AHEAD>
__device__ __forceinline__ float4 volume_pixel(const RenderArgs& a, const TechArgs& t, const float* s_tf, int px,
                                               int py, uint32_t& samples, uint32_t& hit) {
  float4 dest = make_float4(0.f, 0.f, 0.f, 0.f);
  samples = 0;
  hit = 0;
  float3 pos, dir;
  if (!ray_setup(a, px, py, pos, dir)) return dest;
  hit = 1;
  const uint32_t max_samples = (uint32_t)a.num_iter * (uint32_t)a.num_iter;  // numIterations <= 1024
  while (samples < max_samples) {
    float3 p[AHEAD + 1];
    float4 f[AHEAD];
    float I[AHEAD];
    p[0] = pos;
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      f[j] = Field<ST, FL>::sample(a, p[j]);
      if (LICVOL) I[j] = sample_licvol(t, p[j]);
      p[j + 1] = march(p[j], dir, a.step_size);
    }
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      float4 src;
      if (LICVOL) {
        const float4 tfv = tf_rgba(s_tf, a.tf_index == VVLIC_TF_INDEX_MAGNITUDE ? f[j].w : f[j].z);
        src = shade<false>(a, s_tf, make_float4(0.f, 0.f, 0.f, I[j]), tfv, p[j], dir, f[j]);  // illumLIC
      } else {
        src = make_float4(f[j].x, f[j].y, f[j].z, tf_rgba(s_tf, f[j].w).w);
      }
      ++samples;
      dest = blend(dest, src);
      if (outside_box(a, p[j + 1]) || dest.w > a.alpha_thr || samples >= max_samples) return dest;
    }
    pos = p[AHEAD];
  }
  return dest;
}

template <int ST, int FL, bool LICVOL, int AHEAD>
__global__ void __launch_bounds__(kThreads) volume_kernel(const __grid_constant__ RenderArgs a,
                                                          const __grid_constant__ TechArgs t) {
  __shared__ __align__(16) float s_tf[5 * VVLIC_TF_ENTRIES];
  load_tf(a, s_tf);
  const int px = blockIdx.x * kTileW + (threadIdx.x % kTileW);
  const int py = blockIdx.y * kTileH + (threadIdx.x / kTileW);
  uint32_t samples = 0, hit = 0;
  if (px < a.W && py < a.H) {
    const float4 dest = volume_pixel<ST, FL, LICVOL, AHEAD>(a, t, s_tf, px, py, samples, hit);
    store_pixel(a, px, py, dest, samples);
  }
  flush_counters(a, samples, hit);
}

// LIC intensity at every voxel centre of the LIC volume: lic3d_volume_fragment.glsl:2-21 with
// pos = ((x+.5)/nx, (y+.5)/ny, (z+.5)/nz) * scaleVol (VolumeBuffer::drawSlice).  A warp takes a
// tile of kLicvolTileW x kLicvolTileH voxels in x, y.  On the 512^3 turbulence field (RK4, L = 60 each way)
// the 8x4 tiles took 202.7 ms against 217.9 ms for 32-voxel rows, and two slices per thread 203.3 ms.
#ifndef VVLIC_LICVOL_TILE
#define VVLIC_LICVOL_TILE 1
#endif
#ifndef VVLIC_LICVOL_MIN_BLOCKS
#define VVLIC_LICVOL_MIN_BLOCKS 1
#endif
constexpr int kLicvolTileW = VVLIC_LICVOL_TILE ? 8 : 32, kLicvolTileH = VVLIC_LICVOL_TILE ? 4 : 1;

// warp work items of an nx*ny*nz LIC volume
__host__ __device__ inline size_t licvol_items(const int ln[3]) {
  return (size_t)((ln[0] + kLicvolTileW - 1) / kLicvolTileW) * (size_t)((ln[1] + kLicvolTileH - 1) / kLicvolTileH) *
         (size_t)ln[2];
}

__device__ __forceinline__ float3 licvol_pos(const RenderArgs& a, const TechArgs& t, int x, int y, int z) {
  return mul3(f3(((float)x + 0.5f) / t.ln[0], ((float)y + 0.5f) / t.ln[1], ((float)z + 0.5f) / t.ln[2]),
              f3(a.scale_vol[0], a.scale_vol[1], a.scale_vol[2]));
}

template <int ST, int FL, int NL, int INTEG>
__global__ void __launch_bounds__(kThreads, VVLIC_LICVOL_MIN_BLOCKS) licvolume_kernel(const __grid_constant__ RenderArgs a,
                                                                                      const __grid_constant__ TechArgs t) {
  const int nx = t.ln[0], ny = t.ln[1];
  const int tx = (nx + kLicvolTileW - 1) / kLicvolTileW, ty = (ny + kLicvolTileH - 1) / kLicvolTileH;
  const size_t items = licvol_items(t.ln);
  const int lane = threadIdx.x & 31;
  const size_t stride = (size_t)gridDim.x * (blockDim.x >> 5);
  for (size_t wi = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); wi < items; wi += stride) {
    const int x = (int)(wi % tx) * kLicvolTileW + lane % kLicvolTileW;
    const int y = (int)((wi / tx) % ty) * kLicvolTileH + lane / kLicvolTileW;
    const int z = (int)(wi / ((size_t)tx * ty));
    if (x >= nx || y >= ny) continue;
    const size_t v = ((size_t)z * ny + y) * nx + x;
    const float3 p0 = licvol_pos(a, t, x, y, z);
    const float4 f0 = Field<ST, FL>::sample(a, p0);
    t.licvol_out[v] = compute_lic<ST, FL, NL, INTEG, false>(a, p0, f0).w * a.intensity_scale;
  }
}

template <int ST, int FL, int NL, int INTEG, bool GRAD>
static cudaError_t launch_tech_one(const RenderArgs& a, const TechArgs& t, int num_sms, cudaStream_t s) {
  if (t.technique == VVLIC_TECHNIQUE_LICVOLUME && t.licvol_out) {
    const size_t threads = licvol_items(t.ln) * 32;
    const int blocks = (int)std::min<size_t>((threads + kThreads - 1) / kThreads, (size_t)152 * 64);
    licvolume_kernel<ST, FL, NL, INTEG><<<std::max(1, blocks), kThreads, 0, s>>>(a, t);
    return cudaGetLastError();
  }
  // Slicing frames by W*H pixels on a chip that holds `warps` warps:
  //   fewer than 1.5 pixels per resident lane: groups of eight planes;
  //   more pixels than planes * warps: a lane per pixel.  Its tail, a chain of all planes, is then
  //     short against the whole, and lanes on one plane share more texels than lanes on several;
  //   a lane per pixel also from 8 pixels per warp where half of all samples would end their ray, and from 16 and twice
  //     the planes that an average ray meets where these are at most 24 (thin volumes), since such rays leave most lanes
  //     of a group idle.  Groups / so, 400^2, default TF, unlit, lit: 4 slices of 96^2 0.115 / 0.061 and 0.146 / 0.075 ms, 16 slices
  //     0.134 / 0.074 and 0.154 / 0.098; half of the alphas opaque, 96^3, 0.18 / 0.058 and 0.22 / 0.075, 200^2 0.069 / 0.041 and
  //     0.078 / 0.047;
  //   groups of two planes between.
  // FP16, ms by eight / two / lane per pixel: 800x600 lit, 160^3 1.92 / 1.92 / 2.13; Heun, a plane per texel,
  // 600^2 1.24 / 1.08 / 1.52, 1024^2 3.18 / 2.53 / 2.69, 1600^2 7.26 / 5.52 / 5.36; RK4, 2.5 texels, 300^2
  // 0.40 / 0.43 / 1.10, 600^2 1.08 / 0.89 / 1.06, 1200^2 3.47 / 2.66 / 2.33; 3.3 texels 300^2 0.22 / 0.23 / 0.39,
  // 600^2 0.57 / 0.43 / 0.43, 900^2 1.14 / 0.82 / 0.66.
  const long long pixels = (long long)a.W * a.H, warps = resident_warps(num_sms);
  const double area = std::fabs(t.v[0]) * a.ext[1] * a.ext[2] + std::fabs(t.v[1]) * a.ext[2] * a.ext[0] +
                      std::fabs(t.v[2]) * a.ext[0] * a.ext[1];
  const double planes = (double)a.ext[0] * a.ext[1] * a.ext[2] / area / t.depth * t.nslices;
  const bool few = planes <= 24.0 && pixels >= std::max(16.0, 2.0 * planes) * warps;
  const bool end = a.end_share >= 0.5f && a.alpha_thr >= 0.95f && pixels >= 8 * warps;
  if ((pixels >= 48 * warps && pixels >= t.nslices * warps) || few || end) {
    const dim3 tiles((a.W + kTileW - 1) / kTileW, (a.H + kTileH - 1) / kTileH);
    slicing_pixel_kernel<ST, FL, NL, INTEG, GRAD><<<tiles, kThreads, 0, s>>>(a, t);
    return cudaGetLastError();
  }
  const int threads = cast_cta_threads<INTEG, GRAD>(a, num_sms);
  const CtaShape cta = cta_shape(threads);
  const auto grid = [&](int tw, int th) {
    return dim3((unsigned)((a.W + tw * cta.wx - 1) / (tw * cta.wx)), (unsigned)((a.H + th * cta.wy - 1) / (th * cta.wy)));
  };
  if (pixels < 48 * warps)
    slicing_kernel<ST, FL, NL, INTEG, GRAD, 8><<<grid(GroupTile<8>::w, GroupTile<8>::h), threads, 0, s>>>(a, t);
  else
    slicing_kernel<ST, FL, NL, INTEG, GRAD, 2><<<grid(GroupTile<2>::w, GroupTile<2>::h), threads, 0, s>>>(a, t);
  return cudaGetLastError();
}

template <int ST, int FL, int NL>
static cudaError_t launch_tech_layout(const RenderArgs& a, const TechArgs& t, int integ, bool grad, int num_sms,
                                      cudaStream_t s) {
  if (t.technique != VVLIC_TECHNIQUE_SLICING && !t.licvol_out) {
    const dim3 grid((a.W + kTileW - 1) / kTileW, (a.H + kTileH - 1) / kTileH);
    // Two samples in flight where half of all samples would end their ray, or rays have up to eight: 2000^2 frame, all
    // opaque 182 -> 153 us, four slices of 96^2 134 -> 109 and, rays that go on, 210 -> 172 (one at a time 152, 108, 173).
    if (t.technique != VVLIC_TECHNIQUE_LICVOLUME) volume_kernel<ST, FL, false, 1><<<grid, kThreads, 0, s>>>(a, t);
    else if (a.end_share >= 0.5f || a.mean_samples <= 8.0f) volume_kernel<ST, FL, true, 2><<<grid, kThreads, 0, s>>>(a, t);
    else volume_kernel<ST, FL, true, 4><<<grid, kThreads, 0, s>>>(a, t);
    return cudaGetLastError();
  }
  if (grad) {
    if (integ == VVLIC_EULER) return launch_tech_one<ST, FL, NL, VVLIC_EULER, true>(a, t, num_sms, s);
    if (integ == VVLIC_HEUN) return launch_tech_one<ST, FL, NL, VVLIC_HEUN, true>(a, t, num_sms, s);
    return launch_tech_one<ST, FL, NL, VVLIC_RK4, true>(a, t, num_sms, s);
  }
  if (integ == VVLIC_EULER) return launch_tech_one<ST, FL, NL, VVLIC_EULER, false>(a, t, num_sms, s);
  if (integ == VVLIC_HEUN) return launch_tech_one<ST, FL, NL, VVLIC_HEUN, false>(a, t, num_sms, s);
  return launch_tech_one<ST, FL, NL, VVLIC_RK4, false>(a, t, num_sms, s);
}

template <int ST>
static cudaError_t launch_tech_storage(const RenderArgs& a, const TechArgs& t, int sampler, int integ, bool grad,
                                       int num_sms, cudaStream_t s) {
  switch (sampler) {
    case VVLIC_SAMPLER_GATHER: return launch_tech_layout<ST, kGather, kGather>(a, t, integ, grad, num_sms, s);
    case VVLIC_SAMPLER_CELL: return launch_tech_layout<ST, kCell, kCell>(a, t, integ, grad, num_sms, s);
    case VVLIC_SAMPLER_TEXTURE:
      if constexpr (ST == VVLIC_STORAGE_BF16) return cudaErrorNotSupported;  // runs as F16 (kernel_storage)
      else return launch_tech_layout<ST, kTexture, kTexture>(a, t, integ, grad, num_sms, s);
    case VVLIC_SAMPLER_HYBRID:
      if constexpr (ST == VVLIC_STORAGE_BF16) return cudaErrorNotSupported;
      else return launch_tech_layout<ST, kTexture, kCellFast>(a, t, integ, grad, num_sms, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vvlic
