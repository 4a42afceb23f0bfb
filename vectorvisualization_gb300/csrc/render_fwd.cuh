// Forward LIC ray-cast kernels: the lic3d_fragment.glsl main() (lic3d_fragment.glsl:5-99) on a raster
// grid of small CTAs, each warp on a tile of rays with S consecutive samples of each side by side
// (trace_group); frames whose rays may end early or are short take one lane to a ray first (head_samples).
// Instantiated per field storage in render_f32.cu / render_f16.cu /
// render_bf16.cu / render_u8.cu so the translation units compile in parallel.
//
// The raster grid took the place of persistent warps that pulled 8x4-pixel tiles longest ray first
// and of a static grid of 16x8-pixel CTAs.  With S = 8 the items are so short that the order no
// longer matters for the tail, and neighbouring rays that run on one SM at a time share texels and
// cells in its L1.  Queue -> raster, both with groups: lit 1024^2 Heun frame of 256^3 60.8 -> 57.7 ms
// (FP32 at 512^2 30.9 -> 27.3), unlit 853x481 frame 2.82 -> 2.68 ms, 128^2 preview 348 -> 190 us.
#pragma once

#include "vvlic_device.cuh"
#include "vvlic_launch.hpp"

namespace vvlic {

constexpr int kTileW = 16, kTileH = 8;         // techniques.cuh: one CTA of 128 threads per tile
constexpr int kThreads = 128, kWarps = kThreads / 32;

// Registers: the ray-cast kernels are compiled for at most 65536 / (128 * VVLIC_MIN_BLOCKS) registers
// per thread and launched in CTAs of up to cast_threads() threads.  Euler and Heun at 7 / 6 / 5, groups of
// four: 512^2 lit frame of 256^3 17.9 / 17.7 / 17.3 ms, 1024^2 61.1 / 60.9 / 62.7 ms, FP32 31.9 / 30.9 /
// 30.0 ms, unlit 853x481 UNORM8 frame 2.90 / 2.79 / 2.78 ms.  RK4 (four slopes per step), 1024^2 frame
// of the lit 512^3 orbit, at 6 / 5 / 4: 488 / 474 / 482 ms.
#ifndef VVLIC_MIN_BLOCKS
#define VVLIC_MIN_BLOCKS 6
#endif
#ifndef VVLIC_RK4_MIN_BLOCKS
#define VVLIC_RK4_MIN_BLOCKS 5
#endif
template <int INTEG> __host__ __device__ constexpr int min_blocks() {
  return INTEG == VVLIC_RK4 ? VVLIC_RK4_MIN_BLOCKS : VVLIC_MIN_BLOCKS;
}
// Lit FP32 kernels take two texture fetches and a 32-byte cell per evaluation: up to 128 registers (2 CTAs of
// 256 threads per SM) against 80, 256^3 frame at 128^2 / 256^2 / 512^2 / 1024^2 4.07 / 8.89 / 26.4 / 93.8 against
// 3.94 / 9.65 / 27.3 / 93.7 ms, Euler at 512^2 15.9 against 16.6.  Unlit ones lose on small frames (128^2
// preview 214 against 188 us, 256^2 Euler 1447 against 1428) what they gain on a 512^2 one (30.1 against 32.6 ms).
template <int INTEG> __host__ __device__ constexpr int cast_threads() { return INTEG == VVLIC_RK4 ? 128 : 256; }
template <int ST, int INTEG, bool GRAD> __host__ __device__ constexpr int cast_min_ctas() {
  return ST == VVLIC_STORAGE_F32 && GRAD && INTEG != VVLIC_RK4 ? 2 : min_blocks<INTEG>() * 128 / cast_threads<INTEG>();
}

__device__ __forceinline__ void load_tf(const RenderArgs& a, float* s_tf) {
  for (int i = threadIdx.x; i < 5 * VVLIC_TF_ENTRIES; i += blockDim.x) s_tf[i] = __ldg(a.tf + i);
  __syncthreads();
}

__device__ __forceinline__ void store_pixel(const RenderArgs& a, int px, int py, float4 dest, uint32_t samples) {
  const size_t pix = (size_t)py * a.W + px;
  if (!in_range(a, (long long)pix, (long long)a.W * a.H, VVLIC_CHECK_IMAGE)) return;
  reinterpret_cast<float4*>(a.out)[pix] = dest;
  if (a.samples) a.samples[pix] = samples;
  if (a.tape_n) {
    a.tape_n[pix] = samples;
    if (samples > (uint32_t)a.tape_stride) atomicAdd(a.tape_overflow, 1ull);  // tape too short
  }
}

__device__ __forceinline__ void flush_counters(const RenderArgs& a, uint32_t samples, uint32_t hits) {
  unsigned s = __reduce_add_sync(0xffffffffu, samples);
  unsigned h = __reduce_add_sync(0xffffffffu, hits);
  if ((threadIdx.x & 31) == 0) {
    if (s) atomicAdd(a.counters + 0, (unsigned long long)s);
    if (s && a.count_steps) atomicAdd(a.counters + 2, (unsigned long long)s * (unsigned)(a.lb + a.lf));
    if (h) atomicAdd(a.counters + 1, (unsigned long long)h);
  }
}

// Rays of a warp: 32 / S as 2x1, 2x2, 4x2 or 4x4 pixels.
template <int S> struct GroupTile {
  static constexpr int w = S >= 8 ? 2 : 4, h = 32 / S / w;
};
struct CtaShape {
  int wx, wy;  // warps across and up
};
__host__ __device__ inline CtaShape cta_shape(int threads) {
  return threads >= 128 ? CtaShape{2, threads / 64} : CtaShape{1, threads / 32};
}

// Which part of its rays a kernel marches: all of it, the first `bound` passes (rays that go on leave the
// composite so far in their pixel, with the sign of alpha set), or the rest of those, behind `bound` samples.
enum Part : int { kWhole, kHead, kRest };

template <int ST, int FL, int NL, int INTEG, bool GRAD, int S, int PART>
__global__ void __launch_bounds__(cast_threads<INTEG>(), cast_min_ctas<ST, INTEG, GRAD>())
    raycast_kernel(const __grid_constant__ RenderArgs a, int strip, uint32_t bound) {
  __shared__ __align__(16) float s_tf[5 * VVLIC_TF_ENTRIES];
  using T = GroupTile<S>;
  if (PART != kRest) load_tf(a, s_tf);
  const CtaShape cta = cta_shape(blockDim.x);
  unsigned bx = blockIdx.x, by = blockIdx.y;
  if (strip) {  // CTAs run up one strip of `strip` columns after the other
    const unsigned i = by * gridDim.x + bx, col = i / (strip * gridDim.y) * strip, rest = i - col * gridDim.y;
    const unsigned width = min((unsigned)strip, gridDim.x - col);
    bx = col + rest % width;
    by = rest / width;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane % (32 / S);
  const int px = ((int)bx * cta.wx + warp % cta.wx) * T::w + r % T::w;
  const int py = ((int)by * cta.wy + warp / cta.wx) * T::h + r / T::w;
  bool ray = px < a.W && py < a.H, open;
  uint32_t samples, hit;
  float4 dest = make_float4(0.f, 0.f, 0.f, 0.f);
  float4* pixel = reinterpret_cast<float4*>(a.out) + ((size_t)py * a.W + px);
  if (PART == kRest) {
    if (ray) {
      dest = *pixel;
      ray = signbit(dest.w);
      dest.w = fabsf(dest.w);
    }
    if (!__syncthreads_or(ray)) return;
    load_tf(a, s_tf);
  }
  dest = trace_group<ST, FL, NL, INTEG, GRAD, S>(a, s_tf, ray, px, py, samples, hit, PART == kRest ? bound : 0u, dest,
                                                 PART == kHead ? bound : 0xffffffffu, open);
  const bool store = ray && lane < 32 / S;
  if (store) {
    if (PART == kHead && open) *pixel = make_float4(dest.x, dest.y, dest.z, -dest.w);
    else store_pixel(a, px, py, dest, samples);
  }
  flush_counters(a, store ? samples - (PART == kRest ? bound : 0u) : 0u, store && PART != kRest ? hit : 0u);
}

// CTA and group size by the number of 2x2-ray warp tiles against the warps the chip holds:
//   fewer tiles than half of them: 16 samples at a time (2x1 rays), the 64^2 preview of a 64^3 field
//     85 us against 125;
//   up to twice as many: 64-thread CTAs, which spread over the SMs more evenly (128^2 preview 189 us
//     against 203 in 128 threads and 234 in 256);
//   from 8 times as many, lit Euler and Heun kernels of the narrower texels: four samples of 4x2 rays,
//     which stay closer together where samples are further apart than pixels: 3.3 texels between samples, 600^2
//     5.01 -> 4.83 ms, 1200^2 16.8 -> 16.2; one texel, 1024^2 57.46 -> 57.44.  (FP32 27.2 -> 28.5, RK4
//     446 -> 465; unlit 14.0 -> 13.6 with coarse samples, but 853x481 UNORM8 2.68 -> 2.79.)
//   from 16 times as many, lit Euler and Heun kernels: 256-thread CTAs, whose 4x8 rays share more noise
//     cells in L1 (FP32 512^2 lit frame 27.3 ms against 29.1; FP16 1024^2 57.7 against 58.9); the unlit ones
//     read a quarter of the cell bytes and lose 1 % by it;
//   128 threads otherwise.
// RK4 grids run up strips of 16 CTAs, so that the rays in flight are a block of the image and not a
// few rows: 2048^2 orbit frame 1379 against 1404 ms, 1024^2 447 against 453 (Heun: 59.6 against 58.9).
inline long long cast_tiles(const RenderArgs& a) { return (long long)((a.W + 1) / 2) * ((a.H + 1) / 2); }
inline long long resident_warps(int num_sms) { return 24ll * num_sms; }
// Samples that a frame's rays take one at a time, a lane to a ray, before the groups: where rays end after a sample
// or two, or are no longer than that, seven of a group's eight lanes are lost.
//   Frames all of whose samples end their ray (end_share 1): all of them, 0xffffffff.
//   Frames whose rays may well end early (may_end): the first 1 to 16 by the frame's size, since a lane to a ray is
//     as fast as groups on a large frame only (192^3, 131 samples a ray, ms by lane / groups: 256^2
//     3.9 / 1.6, 512^2 6.6 / 5.2, 1024^2 19.4 / 19.3).  All opaque, 1024^2, groups alone / so: unlit 1.23 / 0.23 ms, lit
//     0.80 / 0.24, FP32 2.24 / 0.40, RK4 2.21 / 0.39.  Rays that go on pay 1 to 3 % for it.
//   Frames of short rays, up to 1.5 times as many samples on average (thin volumes): all of them, 0xffffffff.
//     512 x 512 x 1 volume, 2 samples a ray, 1024^2, groups / so: unlit 1.13 / 0.31 ms, lit 0.81 / 0.40, RK4 1.97 / 0.56;
//     14 samples a ray 2.42 / 2.07, 3.08 / 2.61, 4.46 / 3.96.
// A recording's checkpoints hold the state before every 32nd sample, which a group knows for its first one only:
// its rays take eight or sixteen samples first, or none where the frame is so small that eight cost 10 %.
inline bool may_end(const RenderArgs& a) { return a.end_share >= 1.0f / 64.0f; }
inline uint32_t head_samples(const RenderArgs& a, int num_sms) {
  if (a.end_share >= 1.0f) return 0xffffffffu;
  const uint32_t head = (uint32_t)std::min<long long>(16, cast_tiles(a) / (2 * resident_warps(num_sms)));
  if (head > 0 && a.mean_samples <= 1.5f * head) return 0xffffffffu;
  return !may_end(a) ? 0u : (a.tape_is ? (head < 3 ? 0u : (head + 7) / 8 * 8) : head);
}
static_assert(kSegment % 8 == 0, "checkpoints at the first sample of a group");
template <int INTEG, bool GRAD> static int cast_cta_threads(const RenderArgs& a, int num_sms) {
  const long long tiles = cast_tiles(a), resident = resident_warps(num_sms);
  return tiles <= 2 * resident ? 64 : (GRAD && INTEG != VVLIC_RK4 && tiles >= 16 * resident ? 256 : 128);
}

// One part of a frame in groups of S samples.
template <int ST, int FL, int NL, int INTEG, bool GRAD, int S, int PART>
static cudaError_t launch_part(const RenderArgs& a, uint32_t bound, int num_sms, cudaStream_t stream) {
  const int threads = cast_cta_threads<INTEG, GRAD>(a, num_sms);
  const int strip = INTEG == VVLIC_RK4 ? 16 : 0;
  const CtaShape cta = cta_shape(threads);
  const int w = GroupTile<S>::w * cta.wx, h = GroupTile<S>::h * cta.wy;
  const dim3 grid((unsigned)((a.W + w - 1) / w), (unsigned)((a.H + h - 1) / h));
  raycast_kernel<ST, FL, NL, INTEG, GRAD, S, PART><<<grid, threads, 0, stream>>>(a, strip, bound);
  return cudaGetLastError();
}

template <int ST, int FL, int NL, int INTEG, bool GRAD>
static cudaError_t launch_one(const RenderArgs& a, int num_sms, cudaStream_t stream) {
  constexpr bool kFours = GRAD && ST != VVLIC_STORAGE_F32 && INTEG != VVLIC_RK4;
  const bool fours = cast_tiles(a) >= 8 * resident_warps(num_sms);
  const uint32_t head = head_samples(a, num_sms);
  if (head > 0) {
    const cudaError_t e = launch_part<ST, FL, NL, INTEG, GRAD, 1, kHead>(a, head, num_sms, stream);
    if (e != cudaSuccess || head == 0xffffffffu) return e;
    if constexpr (kFours)
      if (fours) return launch_part<ST, FL, NL, INTEG, GRAD, 4, kRest>(a, head, num_sms, stream);
    return launch_part<ST, FL, NL, INTEG, GRAD, 8, kRest>(a, head, num_sms, stream);
  }
  if constexpr (kFours)
    if (fours) return launch_part<ST, FL, NL, INTEG, GRAD, 4, kWhole>(a, 0u, num_sms, stream);
  if (2 * cast_tiles(a) <= resident_warps(num_sms))
    return launch_part<ST, FL, NL, INTEG, GRAD, 16, kWhole>(a, 0u, num_sms, stream);
  return launch_part<ST, FL, NL, INTEG, GRAD, 8, kWhole>(a, 0u, num_sms, stream);
}

template <int ST, int FL, int NL>
static cudaError_t launch_layout(const RenderArgs& a, int integ, bool grad, int num_sms, cudaStream_t s) {
  if (grad) {
    if (integ == VVLIC_EULER) return launch_one<ST, FL, NL, VVLIC_EULER, true>(a, num_sms, s);
    if (integ == VVLIC_HEUN) return launch_one<ST, FL, NL, VVLIC_HEUN, true>(a, num_sms, s);
    return launch_one<ST, FL, NL, VVLIC_RK4, true>(a, num_sms, s);
  }
  if (integ == VVLIC_EULER) return launch_one<ST, FL, NL, VVLIC_EULER, false>(a, num_sms, s);
  if (integ == VVLIC_HEUN) return launch_one<ST, FL, NL, VVLIC_HEUN, false>(a, num_sms, s);
  return launch_one<ST, FL, NL, VVLIC_RK4, false>(a, num_sms, s);
}

// Sampler (VVLIC_SAMPLER_*) -> (field layout, noise layout).
template <int ST>
static cudaError_t launch_storage(const RenderArgs& a, int sampler, int integ, bool grad, int num_sms, cudaStream_t s) {
  switch (sampler) {
    case VVLIC_SAMPLER_GATHER: return launch_layout<ST, kGather, kGather>(a, integ, grad, num_sms, s);
    case VVLIC_SAMPLER_CELL: return launch_layout<ST, kCell, kCell>(a, integ, grad, num_sms, s);
    case VVLIC_SAMPLER_TEXTURE:
      if constexpr (ST == VVLIC_STORAGE_BF16) return cudaErrorNotSupported;  // runs as F16 (kernel_storage)
      else return launch_layout<ST, kTexture, kTexture>(a, integ, grad, num_sms, s);
    case VVLIC_SAMPLER_HYBRID:
      if constexpr (ST == VVLIC_STORAGE_BF16) return cudaErrorNotSupported;
      else return launch_layout<ST, kTexture, kCellFast>(a, integ, grad, num_sms, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vvlic
