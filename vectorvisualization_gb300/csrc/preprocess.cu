// Device preprocessing: field encoding (dataset.cpp:533-635), noise gradients
// (gradient.cpp:190-531 + dataset.cpp:1270-1286) and the corner-packed cell arrays.
//
// This file is compiled with -fmad=false: every float expression rounds like the reference's
// CPU code (no fused multiply-add), so the encoded field and the quantised gradients are
// bit-identical to the reference's own arithmetic.  The one explicit fma (quantize_unit) only
// decides a byte where it provably equals the reference's double expression.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "../../include/vvlic.h"
#include "vvlic_device.cuh"
#include "vvlic_launch.hpp"

namespace vvlic {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float vlen_f32(const float* f) { return sqrtf(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]); }

// Magnitude of voxel a as fillTexDataFloatInterp computes it (0 below EPS = 1e-5f).
__device__ __forceinline__ float voxel_len(const void* xyz, int dtype, size_t a, unsigned char t[3]) {
  float len;
  if (dtype == VVLIC_DTYPE_UINT8) {
    const uint8_t* u = reinterpret_cast<const uint8_t*>(xyz) + 3 * a;
    // `dataU -= 128` on unsigned char wraps modulo 256 (dataset.cpp:565-569)
    for (int c = 0; c < 3; ++c) t[c] = (unsigned char)(u[c] - 128);
    len = sqrtf((float)((int)t[0] * t[0]) + (float)((int)t[1] * t[1]) + (float)((int)t[2] * t[2]));
  } else {
    len = vlen_f32(reinterpret_cast<const float*>(xyz) + 3 * a);
  }
  return len < 1e-5f ? 0.0f : len;
}

// The largest magnitude of the field: four FP32 vectors per thread and iteration in three 16-byte
// loads (VEC: 16-byte aligned input), one atomicMax per CTA.  Bound by memory; one atomic per warp on
// the single word cost 46 us on a 128^3 field whose vectors take 12 us to read.
template <bool VEC> __global__ void field_maxlen_kernel(const void* xyz, int dtype, size_t count, unsigned* maxbits) {
  float m = 0.0f;
  const size_t first = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  size_t rest = 0;
  if (VEC) {
    const float4* q = reinterpret_cast<const float4*>(xyz);
    for (size_t g = first; g < count / 4; g += step) {
      const float4 a = __ldg(q + 3 * g), b = __ldg(q + 3 * g + 1), c = __ldg(q + 3 * g + 2);
      const float v[4][3] = {{a.x, a.y, a.z}, {a.w, b.x, b.y}, {b.z, b.w, c.x}, {c.y, c.z, c.w}};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float len = vlen_f32(v[i]);
        m = fmaxf(m, len < 1e-5f ? 0.0f : len);
      }
    }
    rest = count / 4 * 4;
  }
  for (size_t a = rest + first; a < count; a += step) {
    unsigned char t[3];
    m = fmaxf(m, voxel_len(xyz, dtype, a, t));
  }
  // non-negative floats order like their bit patterns
  __shared__ unsigned s_max[kThreads / 32];
  const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = w;
  __syncthreads();
  if (threadIdx.x < 32) {
    const unsigned b = __reduce_max_sync(0xffffffffu, threadIdx.x < kThreads / 32 ? s_max[threadIdx.x] : 0u);
    if (threadIdx.x == 0) atomicMax(maxbits, b);
  }
}

// The machine word(s) of one texel.
template <int ST> struct TexelWord {
  using type = typename std::conditional<ST == VVLIC_STORAGE_F32, float4,
                                         typename std::conditional<ST == VVLIC_STORAGE_UNORM8, uint32_t, uint2>::type>::type;
};

template <int ST>
__device__ __forceinline__ typename TexelWord<ST>::type encode_texel(float r, float g, float b, float al) {
  if constexpr (ST == VVLIC_STORAGE_F32) {
    return make_float4(r, g, b, al);
  } else if constexpr (ST == VVLIC_STORAGE_F16) {
    __half2 lo = __halves2half2(__float2half_rn(r), __float2half_rn(g));
    __half2 hi = __halves2half2(__float2half_rn(b), __float2half_rn(al));
    uint2 v;
    v.x = *reinterpret_cast<unsigned*>(&lo);
    v.y = *reinterpret_cast<unsigned*>(&hi);
    return v;
  } else if constexpr (ST == VVLIC_STORAGE_UNORM8) {
    // nearest multiple of 1/255 (x*255 rounded in float, then to nearest integer)
    const unsigned q0 = __float2uint_rn(r * 255.0f), q1 = __float2uint_rn(g * 255.0f),
                   q2 = __float2uint_rn(b * 255.0f), q3 = __float2uint_rn(al * 255.0f);
    return min(q0, 255u) | (min(q1, 255u) << 8) | (min(q2, 255u) << 16) | (min(q3, 255u) << 24);
  } else {
    __nv_bfloat16 br = __float2bfloat16_rn(r), bg = __float2bfloat16_rn(g), bb = __float2bfloat16_rn(b),
                  ba = __float2bfloat16_rn(al);
    uint2 v;
    v.x = (unsigned)*reinterpret_cast<unsigned short*>(&br) | ((unsigned)*reinterpret_cast<unsigned short*>(&bg) << 16);
    v.y = (unsigned)*reinterpret_cast<unsigned short*>(&bb) | ((unsigned)*reinterpret_cast<unsigned short*>(&ba) << 16);
    return v;
  }
}

// Voxel tiles of the kernels that write texture arrays: a CTA takes 32 x 8 voxels of kTileZ slices, a warp
// 8 x 4 of them, so that its writes of 8-byte texels fill 64-byte rows of the arrays' block-linear
// tiles next to one another.  Bound by memory: 5.8 TB/s of DRAM traffic in the encode, 6.4 in the
// maximum pass.  512^3 half4 field update and its frame: 1612 us with the arrays filled from the texels,
// 1322 us filled by an encode in rows of 32 voxels, 960 us so (one slice per thread 1082, four 967).
constexpr int kTileZ = 8;
inline dim3 tile_grid(const int n[3]) {
  return dim3((unsigned)((n[0] + 31) / 32), (unsigned)((n[1] + 7) / 8), (unsigned)((n[2] + kTileZ - 1) / kTileZ));
}
__device__ __forceinline__ bool tile_voxel(int nx, int ny, int& x, int& y) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  x = (int)blockIdx.x * 32 + (warp & 3) * 8 + (lane & 7);
  y = (int)blockIdx.y * 8 + (warp >> 2) * 4 + (lane >> 3);
  return x < nx && y < ny;
}

// The texel of voxel (x, y, z) into the volume's texture arrays.
template <int ST>
__device__ __forceinline__ void store_array(const FieldSurfaces& s, int x, int y, int z,
                                            typename TexelWord<ST>::type t) {
  if constexpr (ST == VVLIC_STORAGE_F32) {
    surf3Dwrite(make_float2(t.x, t.y), s.rgba, x * 8, y, z);
    surf3Dwrite(t.z, s.z, x * 4, y, z);
    surf3Dwrite(t.w, s.w, x * 4, y, z);
  } else if constexpr (ST == VVLIC_STORAGE_BF16) {
    const __half2 lo = __floats2half2_rn(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xffff0000u));
    const __half2 hi = __floats2half2_rn(__uint_as_float(t.y << 16), __uint_as_float(t.y & 0xffff0000u));
    surf3Dwrite(make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi)), s.rgba,
                x * 8, y, z);
  } else if constexpr (ST == VVLIC_STORAGE_F16) {
    surf3Dwrite(t, s.rgba, x * 8, y, z);
  } else {
    surf3Dwrite(t, s.rgba, x * 4, y, z);
  }
}


// The encoded texel of voxel a (fillTexDataFloatInterp).
template <int ST>
__device__ __forceinline__ typename TexelWord<ST>::type encode_voxel(const void* xyz, int dtype, size_t a, float max_len) {
  unsigned char t[3];
  float len = voxel_len(xyz, dtype, a, t);
  float r, g, b;
  if (len == 0.0f) {
    r = g = b = 0.5f;
  } else if (dtype == VVLIC_DTYPE_UINT8) {
    r = 0.5f * (float)t[0] / len + 0.5f;
    g = 0.5f * (float)t[1] / len + 0.5f;
    b = 0.5f * (float)t[2] / len + 0.5f;
  } else {
    const float* f = reinterpret_cast<const float*>(xyz) + 3 * a;
    r = 0.5f * f[0] / len + 0.5f;
    g = 0.5f * f[1] / len + 0.5f;
    b = 0.5f * f[2] / len + 0.5f;
  }
  float al = max_len > 0.0f ? len / max_len : 0.0f;
  al = (al > 1.0f) ? 1.0f : ((al < 0.0f) ? 0.0f : al);
  return encode_texel<ST>(r, g, b, al);
}

// Voxels run last to first in both encode kernels: the maximum pass before them left the field's end
// in L2.
template <int ST>
__global__ void field_encode_kernel(const void* xyz, int dtype, size_t count, const unsigned* maxbits, void* out) {
  const float max_len = __uint_as_float(*maxbits);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
    const size_t a = count - 1 - i;
    reinterpret_cast<typename TexelWord<ST>::type*>(out)[a] = encode_voxel<ST>(xyz, dtype, a, max_len);
  }
}

// The same with the volume's texture arrays.
template <int ST>
__global__ void __launch_bounds__(kThreads) field_encode_arrays_kernel(const void* xyz, int dtype, int nx, int ny, int nz,
                                                                       const unsigned* maxbits, void* out,
                                                                       const __grid_constant__ FieldSurfaces arr) {
  const float max_len = __uint_as_float(*maxbits);
  int x, y;
  if (!tile_voxel(nx, ny, x, y)) return;
  const int z1 = nz - (int)blockIdx.z * kTileZ;  // slices z1 - kTileZ .. z1 - 1
#pragma unroll
  for (int i = 1; i <= kTileZ; ++i) {
    const int z = z1 - i;
    if (z < 0) break;
    const size_t a = ((size_t)z * ny + y) * nx + x;
    const auto texel = encode_voxel<ST>(xyz, dtype, a, max_len);
    reinterpret_cast<typename TexelWord<ST>::type*>(out)[a] = texel;
    store_array<ST>(arr, x, y, z, texel);
  }
}

// ------------------------------------------------------------------------------------------
// noise gradients: computeGradients, filterGradients, quantizeGradients and the RGBA pack
// (gradient.cpp:190-531, dataset.cpp:1270-1286) in one pass over the noise
// ------------------------------------------------------------------------------------------
// A CTA owns a 32 x 16 tile of raw gradients and marches it through a run of slices.  A slice's raw
// gradients go to shared memory once, and every voxel adds its nine neighbours of the slice to
// the three windows that contain them (those of voxels z + 2, z + 1 and z), so a raw gradient never
// reaches global memory: 1 byte read and 4 written per voxel remain.  The outputs are the tile
// without its two low rows and columns, the halo the windows read.
//
// Each window's terms are added in the reference's (k, j, i) order with every product and sum
// rounded by itself, as the reference's CPU code does, so the 81 products and 81 sums of a voxel
// cannot be merged into FMAs or into a separable filter; x and y go as packed pairs.  Instruction
// issue is the bound (68 % busy, the FMA pipe 36 %): 430 instructions for a thread's two voxels, a
// quarter of them for the halo.  512^3 central differences 3604 -> 1405 us, Sobel 2000 us, against
// the two passes that wrote and re-read 16 bytes of raw gradient per voxel.
constexpr int kGradTileX = 32, kGradTileY = 16, kGradRows = 2;  // raw gradients per CTA, rows per thread
constexpr int kGradHalo = 2;
constexpr int kGradOutX = kGradTileX - kGradHalo, kGradOutY = kGradTileY - kGradHalo;
constexpr int kGradThreads = kGradTileX * kGradTileY / kGradRows;

struct GradArgs {
  const uint8_t* v;
  uint32_t* out;
  int nx, ny, nz, zrun;  // slices of output per CTA
  float sd[3];
  float w[10];       // window weights by i^2 + j^2 + k^2 (kGradWeight)
  float minus_zero;  // -0.0f (mul_then_add2)
};
// A window weight depends on i^2 + j^2 + k^2 alone (i, j, k in 0..2 from the window's near corner): ten
// values, kept as register pairs; equal products of a gradient are formed once.
__host__ __device__ constexpr int grad_weight(int k, int j, int i) {
  const int d = (2 - k) * (2 - k) + (2 - j) * (2 - j) + (2 - i) * (2 - i);
  return d < 7 ? d : (d == 8 ? 7 : (d == 9 ? 8 : 9));
}

// (unsigned char)(((double)c + 1.0) / 2.0 * 255.0), quantizeGradients' conversion of a unit
// component c (gradient.cpp:466-477), without double arithmetic for almost every input.  The
// float t = fma(c, 127.5, 127.5) is within 2^-17 of the exact (c + 1) * 127.5 and the double
// expression within 2^-44 of it; the exact value is an integer only at c = -1 and c = 1, so
// when t lies more than 1e-4 from an integer both truncate to floor(t).  Inputs nearer an
// integer (about 2 in 10^4) take the double expression itself, in a call of its own so that the
// compiler cannot evaluate it speculatively for every voxel (GB300's FP64 rate is a small
// fraction of its FP32 rate).
__device__ __noinline__ unsigned char quantize_unit_double(float c) {
  return (unsigned char)(((double)c + 1.0) / 2.0 * 255.0);
}
__device__ __forceinline__ unsigned char quantize_unit(float c) {
  const float t = fmaf(c, 127.5f, 127.5f);
  const float f = floorf(t);
  const float r = t - f;
  if (r > 1e-4f && r < 1.0f - 1e-4f) return (unsigned char)(int)f;
  return quantize_unit_double(c);
}

// The window sum's RGBA texel as the reference computes it: length, three divisions and the
// conversion.  In a call of its own: few voxels need it (pack_gradient).
__device__ __noinline__ uint32_t pack_gradient_exact(float x, float y, float z, unsigned value) {
  const float len = sqrtf(x * x + y * y + z * z);
  if (len < 1e-5f) {
    x = y = z = 0.0f;
  } else {
    x /= len;
    y /= len;
    z /= len;
  }
  return (uint32_t)quantize_unit(x) | ((uint32_t)quantize_unit(y) << 8) | ((uint32_t)quantize_unit(z) << 16) |
         (value << 24);
}

// The same texel from one reciprocal square root when no component lies near a step.  With s the
// float sum of squares, t = fma(c * rsqrt(s), 127.5, 127.5) differs from (q + 1) * 127.5 of the
// reference's float quotient q by less than 6.2e-5: rsqrtf is good to 2 ulp, the product, the
// reference's square root and its division to half an ulp each (3.5 * 2^-23 of at most 127.5), and
// the FMA rounds by 2^-17.  Where t lies more than 2e-4 from an integer both truncate alike; about one
// voxel in 800 takes the exact form, and those whose length the 1e-5 cut may decide.
__device__ __forceinline__ uint32_t pack_gradient(float x, float y, float z, unsigned value) {
  const float s = x * x + y * y + z * z;
  const float inv = rsqrtf(s);
  const float tx = fmaf(x * inv, 127.5f, 127.5f), ty = fmaf(y * inv, 127.5f, 127.5f), tz = fmaf(z * inv, 127.5f, 127.5f);
  const float fx = floorf(tx), fy = floorf(ty), fz = floorf(tz);
  const float rx = tx - fx, ry = ty - fy, rz = tz - fz;
  const float lo = fminf(fminf(rx, ry), rz), hi = fmaxf(fmaxf(rx, ry), rz);
  // (comparisons false for NaN)
  if (s > 1e-8f && lo > 2e-4f && hi < 1.0f - 2e-4f)
    return (uint32_t)(int)fx | ((uint32_t)(int)fy << 8) | ((uint32_t)(int)fz << 16) | (value << 24);
  return pack_gradient_exact(x, y, z, value);
}

// acc + w * v per component, the product and the sum each rounded.  The assembler merges a packed
// multiplication and addition into one FMA even in their .rn forms and with -fmad=false (one byte in
// 10^5 came out off by one), so the product is formed as fma(w, v, -0), whose -0 it cannot see.
__device__ __forceinline__ float2 mul_then_add2(float2 w, float2 v, float2 acc, float2 minus_zero) {
  return __fadd2_rn(acc, __ffma2_rn(w, v, minus_zero));
}

// What a noise slice contributes to raw gradients at one voxel: d along x and y, and for SOBEL the
// partial sums of the 3x3x3 masks (gradient.cpp:199-224: weight 1, 3 or 6 by the two axes across,
// 3 times heavier in the derivative's own plane; sums of bytes, exact in float in any order).
template <bool SOBEL> struct GradSlice;
template <> struct GradSlice<false> {
  float c, dx, dy;
};
template <> struct GradSlice<true> {
  float c, x1, x3, y1, y3, s;  // d/dx and d/dy of the (1,3,1) and (3,6,3) sums, sum over the plane
};

// Both rows of a thread in one slice.  v: the slice (the same for the whole CTA); o: 32-bit offsets of the
// row below, the two rows and the row above, each that of the nearest row inside; xm, xp: those of
// the x neighbours (0 outside the volume).  The rows are each other's y neighbours.
template <bool SOBEL>
__device__ __forceinline__ void grad_slices(const uint8_t* v, const unsigned (&o)[4], int xm, int xp,
                                            GradSlice<SOBEL> (&g)[kGradRows]) {
  if constexpr (SOBEL) {
    float n[4][3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      n[i][0] = (float)v[o[i] + xm];
      n[i][1] = (float)v[o[i]];
      n[i][2] = (float)v[o[i] + xp];
    }
#pragma unroll
    for (int q = 0; q < kGradRows; ++q) {
      const float *lo = n[q], *mi = n[q + 1], *hi = n[q + 2];
      g[q].c = mi[1];
      g[q].x1 = (lo[2] - lo[0]) + 3.0f * (mi[2] - mi[0]) + (hi[2] - hi[0]);
      g[q].x3 = 3.0f * (lo[2] - lo[0]) + 6.0f * (mi[2] - mi[0]) + 3.0f * (hi[2] - hi[0]);
      g[q].y1 = (hi[0] - lo[0]) + 3.0f * (hi[1] - lo[1]) + (hi[2] - lo[2]);
      g[q].y3 = 3.0f * (hi[0] - lo[0]) + 6.0f * (hi[1] - lo[1]) + 3.0f * (hi[2] - lo[2]);
      g[q].s = lo[0] + lo[2] + hi[0] + hi[2] + 3.0f * (lo[1] + mi[0] + mi[2] + hi[1]) + 6.0f * mi[1];
    }
  } else {
    g[0].c = (float)v[o[1]];
    g[1].c = (float)v[o[2]];
    g[0].dx = (float)v[o[1] + xp] - (float)v[o[1] + xm];
    g[1].dx = (float)v[o[2] + xp] - (float)v[o[2] + xm];
    g[0].dy = g[1].c - (float)v[o[0]];
    g[1].dy = (float)v[o[3]] - g[0].c;
  }
}

// CTAs per SM: 4 at 64 registers for central differences (512^3 in 1405 us; 3 at 80 registers 1449, 2 at
// 104 1655), 3 for Sobel, whose slices hold twice the values (1995 us against 2415 at 4).
template <bool SOBEL, bool UNIT>
__global__ void __launch_bounds__(kGradThreads, SOBEL ? 3 : 4) noise_gradient_kernel(const __grid_constant__ GradArgs a) {
  // raw gradients of the current and the previous slice, (x, y) pairs and z; a third buffer lets the
  // next slice be written while slower warps still read these (one barrier a slice)
  __shared__ float2 s_xy[3][kGradTileY][kGradTileX];
  __shared__ float s_z[3][kGradTileY][kGradTileX];
  const int tx = threadIdx.x, ty = threadIdx.y * kGradRows;
  const int x = (int)blockIdx.x * kGradOutX - kGradHalo + tx;
  const int y0 = (int)blockIdx.y * kGradOutY - kGradHalo + ty;
  const int z0 = (int)blockIdx.z * a.zrun, z1 = min(z0 + a.zrun, a.nz);
  // voxels outside the volume stand in for the nearest inside; no window reads their gradients
  const int xc = min(max(x, 0), a.nx - 1);
  const int xm = xc > 0 ? -1 : 0, xp = xc < a.nx - 1 ? 1 : 0;
  int yc[4];
  unsigned o[4];  // below, first row, second row, above
  yc[1] = min(max(y0, 0), a.ny - 1);
  yc[2] = min(max(y0 + 1, 0), a.ny - 1);
  yc[0] = max(yc[1] - 1, 0);
  yc[3] = min(yc[2] + 1, a.ny - 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = (unsigned)yc[i] * (unsigned)a.nx + (unsigned)xc;
  const size_t slice = (size_t)a.nx * a.ny;
  const bool writes = tx >= kGradHalo && ty >= kGradHalo;
  int edge[kGradRows];  // distance to the volume's x and y borders, below 0 for rows outside
#pragma unroll
  for (int q = 0; q < kGradRows; ++q) edge[q] = min(min(x, a.nx - 1 - x), min(y0 + q, a.ny - 1 - (y0 + q)));
  const int zs = max(z0 - kGradHalo, 0);
  const float2 zero = make_float2(0.0f, 0.0f), nz = make_float2(a.minus_zero, a.minus_zero);
  float2 w2[10];
#pragma unroll
  for (int i = 0; i < 10; ++i) w2[i] = make_float2(a.w[i], a.w[i]);
  // rings of three, their slots named by the phase (s - zs) % 3 so that nothing is moved: noise
  // slices s - 1, s, s + 1, and the windows of voxels s + 2 (one slice in), s + 1 (two) and s (three)
  GradSlice<SOBEL> ring[3][kGradRows];
  float2 xy[3][kGradRows];
  float zz[3][kGradRows];
  grad_slices<SOBEL>(a.v + max(zs - 1, 0) * slice, o, xm, xp, ring[0]);
  grad_slices<SOBEL>(a.v + zs * slice, o, xm, xp, ring[1]);
  grad_slices<SOBEL>(a.v + min(zs + 1, a.nz - 1) * slice, o, xm, xp, ring[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int q = 0; q < kGradRows; ++q) {
      xy[k][q] = zero;
      zz[k][q] = 0.0f;
    }
  const auto step = [&](auto phase, int s) {
    constexpr int P0 = decltype(phase)::value, P1 = (P0 + 1) % 3, P2 = (P0 + 2) % 3;
    auto &prev = ring[P0], &cur = ring[P1], &next = ring[P2];
    GradSlice<SOBEL> ahead[kGradRows];  // two slices on, so that its loads have a slice's time
    grad_slices<SOBEL>(a.v + min(s + 2, a.nz - 1) * slice, o, xm, xp, ahead);
#pragma unroll
    for (int q = 0; q < kGradRows; ++q) {
      // computeGradients (gradient.cpp:190-374): the Sobel sum inside, one-sided differences on its
      // border; central differences (SOBEL 0), one-sided on the border
      float g[3];
      const int P[3] = {xc, yc[1 + q], s}, N[3] = {a.nx, a.ny, a.nz};
      if constexpr (SOBEL) {
        const bool inside = xc > 0 && xc < a.nx - 1 && yc[1 + q] > 0 && yc[1 + q] < a.ny - 1 && s > 0 && s < a.nz - 1;
        if (inside) {
          g[0] = prev[q].x1 + cur[q].x3 + next[q].x1;
          g[1] = prev[q].y1 + cur[q].y3 + next[q].y1;
          g[2] = next[q].s - prev[q].s;
#pragma unroll
          for (int d = 0; d < 3; ++d) g[d] = UNIT ? g[d] * 0.5f : g[d] / (2.0f * a.sd[d]);
        } else {
          const uint8_t* cp = a.v + s * slice + o[1 + q];
          const size_t st[3] = {1, (size_t)a.nx, slice};
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            g[d] = P[d] >= 1 ? cur[q].c - (float)*(cp - st[d]) : (N[d] > 1 ? (float)cp[st[d]] - cur[q].c : 0.0f);
            if (!UNIT) g[d] = g[d] / a.sd[d];
          }
        }
      } else {
        // outside neighbours stand in for the voxel itself: the difference is the one-sided one
        g[0] = cur[q].dx;
        g[1] = cur[q].dy;
        g[2] = next[q].c - (s > 0 ? prev[q].c : cur[q].c);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (!UNIT) g[d] = g[d] / a.sd[d];
          if (P[d] >= 1 && P[d] < N[d] - 1) g[d] = g[d] * 0.5f;
        }
      }
      s_xy[P0][ty + q][tx] = make_float2(g[0], g[1]);
      s_z[P0][ty + q][tx] = g[2];
      prev[q] = ahead[q];
    }
    __syncthreads();
    if (!writes) return;
    // rows ty - 2 .. ty + 1 of the slice: row r is window row j = r - q of output row q.  Slots: the
    // window one slice in is in P2, two in P1, three (finished here) in P0.
#pragma unroll
    for (int r = 0; r < kGradRows + 2; ++r) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float2 gxy = s_xy[P0][ty - 2 + r][tx - 2 + i];
        const float gz = s_z[P0][ty - 2 + r][tx - 2 + i];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int slot = k == 0 ? P2 : (k == 1 ? P1 : P0);
#pragma unroll
          for (int q = 0; q < kGradRows; ++q) {
            if (r < q || r - q > 2) continue;
            const int w = grad_weight(k, r - q, i);
            xy[slot][q] = mul_then_add2(w2[w], gxy, xy[slot][q], nz);
            zz[slot][q] = __fadd_rn(zz[slot][q], __fmul_rn(a.w[w], gz));
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kGradRows; ++q) {
      if (s >= z0 && edge[q] >= 0) {
        // filterGradients' window shrinks towards the border (gradient.cpp:423-444): whole from two
        // voxels in, its far corner one voxel in, empty on the border
        const int bd = min(edge[q], min(s, a.nz - 1 - s));
        float ax = xy[P0][q].x, ay = xy[P0][q].y, az = zz[P0][q];
        if (bd < 2) {
          ax = ay = az = 0.0f;
          if (bd == 1) {
            const float2 c = s_xy[P2][ty + q - 1][tx - 1];
            ax = a.w[9] * c.x;
            ay = a.w[9] * c.y;
            az = a.w[9] * s_z[P2][ty + q - 1][tx - 1];
          }
        }
        (a.out + s * slice)[o[1 + q]] = pack_gradient(ax, ay, az, (unsigned)cur[q].c);
      }
      xy[P0][q] = zero;
      zz[P0][q] = 0.0f;
    }
  };
  for (int s = zs; s < z1; s += 3) {
    step(std::integral_constant<int, 0>(), s);
    if (s + 1 < z1) step(std::integral_constant<int, 1>(), s + 1);
    if (s + 2 < z1) step(std::integral_constant<int, 2>(), s + 2);
  }
}

// cell c per axis covers texels clamp(c-1), clamp(c): (n+1)^3 cells of 8 texels
template <int ST>
__global__ void field_cells_kernel(const void* texels, int nx, int ny, int nz, void* cells) {
  using T = typename TexelWord<ST>::type;
  const T* t = reinterpret_cast<const T*>(texels);
  T* c = reinterpret_cast<T*>(cells);
  const int cx = nx + 1, cy = ny + 1, cz = nz + 1;
  const size_t count = (size_t)cx * cy * cz;
  for (size_t a = blockIdx.x * (size_t)blockDim.x + threadIdx.x; a < count; a += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(a % cx), y = (int)((a / cx) % cy), z = (int)(a / ((size_t)cx * cy));
    const int x0 = max(x - 1, 0), x1 = min(x, nx - 1), y0 = max(y - 1, 0), y1 = min(y, ny - 1), z0 = max(z - 1, 0),
              z1 = min(z, nz - 1);
    const int xs[2] = {x0, x1}, ys[2] = {y0, y1}, zs[2] = {z0, z1};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      c[8 * a + k] = t[((size_t)zs[(k >> 2) & 1] * ny + ys[(k >> 1) & 1]) * nx + xs[k & 1]];
    }
  }
}

// noise cell i per axis covers texels i and (i+1) mod m (REPEAT); an axis of one texel has two cells
// (noise_cell_extent)
__global__ void noise_cells_kernel(const uint8_t* texels, int mx, int my, int mz, int ch, uint8_t* cells) {
  const int m[3] = {noise_cell_extent(mx), noise_cell_extent(my), noise_cell_extent(mz)};
  const size_t count = noise_cell_count(m);
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < count; v += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(v % m[0]), y = (int)((v / m[0]) % m[1]), z = (int)(v / ((size_t)m[0] * m[1]));
    const size_t a = noise_cell_index(x, y, z, m);
    const int xs[2] = {x < mx ? x : 0, x + 1 < mx ? x + 1 : 0}, ys[2] = {y < my ? y : 0, y + 1 < my ? y + 1 : 0},
              zs[2] = {z < mz ? z : 0, z + 1 < mz ? z + 1 : 0};
    // the cell is assembled in registers and written with 16-byte (RGBA: 32-byte cells) or one
    // 8-byte (value: 8-byte cells) stores; cells are 32- / 8-byte aligned
    if (ch == 4) {
      const uint32_t* t = reinterpret_cast<const uint32_t*>(texels);
      uint32_t q[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = t[((size_t)zs[(k >> 2) & 1] * my + ys[(k >> 1) & 1]) * mx + xs[k & 1]];
      uint4* c = reinterpret_cast<uint4*>(cells) + 2 * a;
      c[0] = make_uint4(q[0], q[1], q[2], q[3]);
      c[1] = make_uint4(q[4], q[5], q[6], q[7]);
    } else {
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        lo |= (uint32_t)texels[((size_t)zs[(k >> 2) & 1] * my + ys[(k >> 1) & 1]) * mx + xs[k & 1]] << (8 * k);
        hi |= (uint32_t)texels[((size_t)zs[1] * my + ys[(k >> 1) & 1]) * mx + xs[k & 1]] << (8 * k);
      }
      reinterpret_cast<uint2*>(cells)[a] = make_uint2(lo, hi);
    }
  }
}

inline int grid_for(size_t count) {
  size_t b = (count + kThreads - 1) / kThreads;
  return (int)(b < 152 * 64 ? (b == 0 ? 1 : b) : 152 * 64);
}

// Texels -> texture arrays through surface writes (a volume's first TEXTURE or HYBRID render).
template <int ST>
__global__ void __launch_bounds__(kThreads) fill_arrays_kernel(const void* texels, int nx, int ny, int nz,
                                                               const __grid_constant__ FieldSurfaces arr) {
  int x, y;
  if (!tile_voxel(nx, ny, x, y)) return;
  const auto* t = reinterpret_cast<const typename TexelWord<ST>::type*>(texels);
#pragma unroll
  for (int i = 0; i < kTileZ; ++i) {
    const int z = (int)blockIdx.z * kTileZ + i;
    if (z < nz) store_array<ST>(arr, x, y, z, t[((size_t)z * ny + y) * nx + x]);
  }
}

}  // namespace

namespace {
// Time interpolation of fillTexData*Interp (dataset.cpp:555-585): t = interpIndex / InterpSize,
// FLOAT3: data + t * (next - data); UCHAR3: the same on the 128-shifted bytes, stored back
// un-shifted so the encoding's own shift recovers the interpolated value.
__global__ void field_interp_kernel(const void* a0, const void* a1, int dtype, size_t count3, float t, void* out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count3; i += (size_t)gridDim.x * blockDim.x) {
    if (dtype == VVLIC_DTYPE_UINT8) {
      const unsigned char d = (unsigned char)(reinterpret_cast<const uint8_t*>(a0)[i] - 128);
      const unsigned char nx = (unsigned char)(reinterpret_cast<const uint8_t*>(a1)[i] - 128);
      const unsigned char v = (unsigned char)((float)d + t * (float)((int)nx - (int)d));
      reinterpret_cast<uint8_t*>(out)[i] = (uint8_t)(v + 128);
    } else {
      const float d = reinterpret_cast<const float*>(a0)[i], nx = reinterpret_cast<const float*>(a1)[i];
      reinterpret_cast<float*>(out)[i] = d + t * (nx - d);
    }
  }
}
}  // namespace

cudaError_t launch_interp_field(const void* d_a0, const void* d_a1, int dtype, const int n[3], float t, void* d_out,
                                cudaStream_t s) {
  const size_t count3 = (size_t)n[0] * n[1] * n[2] * 3;
  field_interp_kernel<<<grid_for(count3), kThreads, 0, s>>>(d_a0, d_a1, dtype, count3, t, d_out);
  return cudaGetLastError();
}

template <int ST>
static void launch_encode(const void* d_xyz, int dtype, const int n[3], void* d_texels, const unsigned* d_maxbits,
                          const FieldSurfaces* arr, cudaStream_t s) {
  const size_t count = (size_t)n[0] * n[1] * n[2];
  if (arr)
    field_encode_arrays_kernel<ST><<<tile_grid(n), kThreads, 0, s>>>(d_xyz, dtype, n[0], n[1], n[2], d_maxbits, d_texels, *arr);
  else field_encode_kernel<ST><<<grid_for(count), kThreads, 0, s>>>(d_xyz, dtype, count, d_maxbits, d_texels);
}

cudaError_t launch_encode_field(const void* d_xyz, int dtype, const int n[3], int storage, void* d_texels,
                                unsigned* d_maxbits, const FieldSurfaces* arr, cudaStream_t s) {
  const size_t count = (size_t)n[0] * n[1] * n[2];
  cudaError_t e = cudaMemsetAsync(d_maxbits, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  const bool vec = dtype == VVLIC_DTYPE_FLOAT32 && (reinterpret_cast<uintptr_t>(d_xyz) & 15) == 0;
  const int grid = std::min(grid_for(vec ? (count + 3) / 4 : count), 152 * 8);
  if (vec) field_maxlen_kernel<true><<<grid, kThreads, 0, s>>>(d_xyz, dtype, count, d_maxbits);
  else field_maxlen_kernel<false><<<grid, kThreads, 0, s>>>(d_xyz, dtype, count, d_maxbits);
  if (storage == VVLIC_STORAGE_F32) launch_encode<VVLIC_STORAGE_F32>(d_xyz, dtype, n, d_texels, d_maxbits, arr, s);
  else if (storage == VVLIC_STORAGE_F16) launch_encode<VVLIC_STORAGE_F16>(d_xyz, dtype, n, d_texels, d_maxbits, arr, s);
  else if (storage == VVLIC_STORAGE_UNORM8)
    launch_encode<VVLIC_STORAGE_UNORM8>(d_xyz, dtype, n, d_texels, d_maxbits, arr, s);
  else launch_encode<VVLIC_STORAGE_BF16>(d_xyz, dtype, n, d_texels, d_maxbits, arr, s);
  return cudaGetLastError();
}

cudaError_t launch_noise_gradients(const uint8_t* d_noise, const int m[3], int mode, const float sd[3], uint8_t* d_rgba,
                                   const float w27[27], cudaStream_t s) {
  GradArgs a;
  a.v = d_noise;
  a.out = reinterpret_cast<uint32_t*>(d_rgba);
  a.nx = m[0];
  a.ny = m[1];
  a.nz = m[2];
  for (int i = 0; i < 3; ++i) a.sd[i] = sd[i];
  for (int k = 0; k < 3; ++k)
    for (int j = 0; j < 3; ++j)
      for (int i = 0; i < 3; ++i) a.w[grad_weight(k, j, i)] = w27[(k * 3 + j) * 3 + i];
  a.minus_zero = -0.0f;
  const int bx = (m[0] + kGradOutX - 1) / kGradOutX, by = (m[1] + kGradOutY - 1) / kGradOutY;
  // Slices per CTA: two more are computed than written, so long runs, but enough CTAs to fill the
  // chip four times over at three per SM; at most 65535 runs (grid limit).
  const long long ctas = 152 * 12;
  a.zrun = (int)std::min<long long>(std::max<long long>(((long long)m[2] * bx * by + ctas - 1) / ctas, 8), 64);
  a.zrun = std::max(a.zrun, (m[2] + 65534) / 65535);
  const dim3 grid((unsigned)bx, (unsigned)by, (unsigned)((m[2] + a.zrun - 1) / a.zrun));
  const dim3 block(kGradTileX, kGradTileY / kGradRows);
  const bool unit = sd[0] == 1.0f && sd[1] == 1.0f && sd[2] == 1.0f;  // division by 1 is exact: left out
  if (mode == VVLIC_NOISE_GRAD_SOBEL) {
    if (unit) noise_gradient_kernel<true, true><<<grid, block, 0, s>>>(a);
    else noise_gradient_kernel<true, false><<<grid, block, 0, s>>>(a);
  } else {
    if (unit) noise_gradient_kernel<false, true><<<grid, block, 0, s>>>(a);
    else noise_gradient_kernel<false, false><<<grid, block, 0, s>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t launch_build_field_cells(const void* d_texels, const int n[3], int storage, void* d_cells,
                                     cudaStream_t s) {
  const size_t count = (size_t)(n[0] + 1) * (n[1] + 1) * (n[2] + 1);
  if (storage == VVLIC_STORAGE_F32)
    field_cells_kernel<VVLIC_STORAGE_F32><<<grid_for(count), kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], d_cells);
  else if (storage == VVLIC_STORAGE_F16)
    field_cells_kernel<VVLIC_STORAGE_F16><<<grid_for(count), kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], d_cells);
  else if (storage == VVLIC_STORAGE_UNORM8)
    field_cells_kernel<VVLIC_STORAGE_UNORM8><<<grid_for(count), kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], d_cells);
  else
    field_cells_kernel<VVLIC_STORAGE_BF16><<<grid_for(count), kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], d_cells);
  return cudaGetLastError();
}

cudaError_t launch_fill_arrays(const void* d_texels, const int n[3], int storage, const FieldSurfaces& arr,
                               cudaStream_t s) {
  const dim3 g = tile_grid(n);
  if (storage == VVLIC_STORAGE_F32)
    fill_arrays_kernel<VVLIC_STORAGE_F32><<<g, kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], arr);
  else if (storage == VVLIC_STORAGE_F16)
    fill_arrays_kernel<VVLIC_STORAGE_F16><<<g, kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], arr);
  else if (storage == VVLIC_STORAGE_UNORM8)
    fill_arrays_kernel<VVLIC_STORAGE_UNORM8><<<g, kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], arr);
  else fill_arrays_kernel<VVLIC_STORAGE_BF16><<<g, kThreads, 0, s>>>(d_texels, n[0], n[1], n[2], arr);
  return cudaGetLastError();
}

cudaError_t launch_build_noise_cells(const uint8_t* d_texels, const int m[3], int ch, uint8_t* d_cells,
                                     cudaStream_t s) {
  const int cells[3] = {noise_cell_extent(m[0]), noise_cell_extent(m[1]), noise_cell_extent(m[2])};
  const size_t count = noise_cell_count(cells);
  noise_cells_kernel<<<grid_for(count), kThreads, 0, s>>>(d_texels, m[0], m[1], m[2], ch, d_cells);
  return cudaGetLastError();
}

}  // namespace vvlic
