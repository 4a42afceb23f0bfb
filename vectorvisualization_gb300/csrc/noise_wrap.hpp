// Wrap form of the noise cells (NoiseCells in vvlic_device.cuh) and the rule that chooses it per
// launch.  Plain C++, so that a host compiler can test the rule.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define VVLIC_HOST_DEVICE __host__ __device__
#else
#define VVLIC_HOST_DEVICE
#endif

namespace vvlic {

// How a noise cell's index wraps (REPEAT), chosen on the host per launch (choose_noise_wrap):
//   kWrapMask  every extent a power of two: a mask;
//   kWrapMul   other extents: a multiply-high by a host-computed reciprocal;
//   kWrapFar   positions whose noise coordinate may exceed +-2^19: floor, conversion and mask or integer
//              remainder.
// The first two take floor(u) from the rounding of one addition: u + 1.5 * 2^23 rounded down holds
// floor(u) in its low mantissa bits (exact for |u| < 2^22).  FRND and F2I, the direct forms, issue
// at an eighth of the FADD rate (15 against 118 lanes per SM clock, three of each per tap).
enum NoiseWrap : int { kWrapFar = 0, kWrapMask = 1, kWrapMul = 2 };
constexpr float kFloorMagic = 12582912.0f;    // 1.5 * 2^23
constexpr unsigned kFloorBits = 0x4B400000u;  // its bit pattern
constexpr int kWrapReach = 1 << 19;           // |noise coordinate| bound of kWrapMask / kWrapMul

// Extent of the noise cells along an axis of m texels: a single texel is held as two equal cells, so that
// every extent has a multiply-high form (an 800x600 frame with a 200 x 150 x 1 noise took 7.82 ms in the
// general form).
VVLIC_HOST_DEVICE inline int noise_cell_extent(int m) { return m > 1 ? m : 2; }

// Wrap constants of an extent m: `clamp` is the coordinate a NaN position reads, congruent
// to -2^24 modulo m (the lower clamp of the general form) and below every finite coordinate;
// `off` a multiple of m that makes indices non-negative; `mul` = floor(2^32 / m) + 1, whose quotient
// is exact for indices below 2^21 (2^21 * 2048 <= 2^32).
VVLIC_HOST_DEVICE inline void noise_wrap_constants(int m, float* clamp, unsigned* mul, unsigned* off) {
  const int r = (1 << 24) % m;
  *clamp = -(float)(((kWrapReach - r) / m) * m + r);
  *off = (unsigned)(((kWrapReach + m - 1) / m) * m);
  *mul = m > 1 ? (unsigned)(0x100000000ull / (unsigned)m) + 1u : 0u;
}

// The larger of the two; NaN if either is.
inline double larger(double a, double b) { return b > a || b != b ? b : a; }

// Largest |position| a streamline of a ray starts at.  Every sample but a ray's first lies in the box the
// ray marches through, [0, tex_max]; the first one, and the planes of a slicing ray, are o + t d for a t
// of the ray's interval in the object box [0, ext], times scale_vol.  `origin` is the largest |component| of
// a pixel's ray origin, `dir` that of the direction all rays share, or 0 where the rays start no
// earlier than t = 0 (perspective views, whose directions have a unit component along the view axis).
//   Rounding: t and t d are good to a few ulps of (|o| + ext) / d, so a camera far away misses the box's
//   face by 2^-18 of its distance at most.
//   Overflow: t stays below far / dir < 1e35 as long as far < 1e35 dir, so an axis whose own 1 / d overflows
//   (|d| < 2^-128) moves by less than 2^-10.  Otherwise (a direction of denormal components, whose
//   interval may begin at t = -inf) there is no bound.
inline double ray_start_bound(const float ext[3], const float scale_vol[3], const float tex_max[3], double origin,
                              double dir) {
  double start = 0.0, far = 0.0;
  for (int i = 0; i < 3; ++i) far = larger(far, origin + std::fabs((double)ext[i]));
  if (!(far < 1e35 * (dir > 0.0 && dir < 0.5 ? dir : 0.5))) return INFINITY;
  for (int i = 0; i < 3; ++i) {
    const double sv = std::fabs((double)scale_vol[i]);
    start = larger(start, larger((1.0 + 1.0 / 1024.0 + far / 262144.0) * larger((double)ext[i], 1.0) * sv, (double)tex_max[i]));
  }
  return start;
}

// The same for the voxel centres of a LIC volume, (0, 1) * scale_vol.
inline double voxel_start_bound(const float scale_vol[3]) {
  double start = 0.0;
  for (int i = 0; i < 3; ++i) start = larger(start, std::fabs((double)scale_vol[i]));
  return start;
}

// The form for streamlines that start within `start` of the origin and move by at most `reach` along
// an axis, under noise texel scales `nscale` (value taps) and `nscale_grad` (gradient taps) and cell
// extents m: |noise coordinate| is bounded by (start + reach) * scale, with a margin for the
// rounding of the positions.  NaN positions read the clamp.
inline int choose_noise_wrap(double start, double reach, const float nscale[3], const float nscale_grad[3],
                             const int m[3]) {
  double scale = 0.0;
  bool mask = true;
  for (int i = 0; i < 3; ++i) {
    scale = larger(scale, larger(std::fabs((double)nscale[i]), std::fabs((double)nscale_grad[i])));
    mask = mask && (m[i] & (m[i] - 1)) == 0;
  }
  const double bound = 1.01 * (start + reach) * scale + 1.0;
  if (!(bound < (double)(kWrapReach - 4096))) return kWrapFar;  // also for NaN
  return mask ? kWrapMask : kWrapMul;
}

}  // namespace vvlic
