// Adjoint of the LIC ray-cast (any shading model + front-to-back blend) with respect
// to the transfer-function table (256 RGBA), the opacity table (256) and the filter taps.
//
// The forward render records a tape: per sample (intensity I, TF coordinate), with gradient
// lighting also the LIC gradient sum G (4 halves), and every kSegment samples a checkpoint
// (position, dest before the sample).  A warp takes four rays, eight consecutive samples of each
// side by side (the forward's groups; adjoint_ray_kernel 32 rays, a lane each, see lane_per_ray), and walks their segments last to first.  From the
// checkpoint it recomputes the compositing states (cheap: no streamline work), the lanes forming
// the sources and every lane of a ray blending them in order; going back, every lane of a ray carries
// the image cotangent through the blends and each lane keeps what its own sample needs.  The
// samples' cotangents (clamp, blend, alpha correction, opacity lookup, shading, TF lookup) and
// their streamlines are then one lane each: the cotangents of I and G are pushed onto the filter taps by
// walking the streamlines once more (dL/dw_j = sum_k S dL/dI_k n_kj + dL/dG_k . g_kj).
//
// Reductions are deterministic: per-tap sums are formed by fixed-order warp exchanges, and
// every contribution enters 64-bit fixed-point accumulators (scale 2^30) by integer atomics,
// which are associative — so the result does not depend on scheduling.
#pragma once

#include "render_fwd.cuh"

namespace vvlic {

// Minimum resident CTAs per SM requested for the adjoint kernels (register cap 65536 / (128 * n)): 6
// (80 registers).  At 7 / 6 / 5 / 4: four-view fit step of 128^3 43.1 / 42.7 / 44.2 / 48.0 ms; RK4, lit,
// L = 60: 128.2 at 3, 118.7 at 4, 118.0 at 5, 117.4 at 6.
#ifndef VVLIC_ADJ_MIN_BLOCKS
#define VVLIC_ADJ_MIN_BLOCKS 6
#endif

constexpr float kFixedScale = 1073741824.0f;  // 2^30
constexpr int kAccTF = 0, kAccOpac = 4 * VVLIC_TF_ENTRIES, kAccTaps = 5 * VVLIC_TF_ENTRIES;
constexpr int kAccSize = kAccTaps + kMaxTaps;

// Adds v to a 64-bit fixed-point accumulator in shared memory, as two 32-bit atomics: the low word's
// old value tells each addition its own carry, so the sum is the 64-bit one in any order.  (64-bit
// shared atomics are compare-and-swap loops, and neighbouring samples hit the same table entries: fit
// step of four 512^2 views 42.7 ms with them, 38.7 so, 38.1 without any.)  |v| < 1 converts in 32
// bits.
__device__ __forceinline__ void fixed_add(long long* slot, float v) {
  if (v == 0.0f) return;
  const float f = v * kFixedScale;
  const long long q = fabsf(v) < 1.0f ? (long long)__float2int_rn(f) : __float2ll_rn(f);
  const unsigned lo = (unsigned)q;
  unsigned hi = (unsigned)((unsigned long long)q >> 32);
  unsigned* w = reinterpret_cast<unsigned*>(slot);
  hi += atomicAdd(w, lo) + lo < lo ? 1u : 0u;
  if (hi) atomicAdd(w + 1, hi);
}

// Sum over the warp (fixed butterfly order); lane 0 adds it to the block accumulator.
__device__ __forceinline__ void warp_fixed_add(long long* slot, float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) fixed_add(slot, v);
}

// One exchange of a warp reduction of two values: lanes with bit `o` clear keep `a`, the others
// `b`, each plus its partner's.
__device__ __forceinline__ float exchange(float a, float b, int o) {
  const bool lo = ((threadIdx.x & 31) & o) == 0;
  return (lo ? a : b) + __shfl_xor_sync(0xffffffffu, lo ? b : a, o);
}

// Warp sums of the tap contributions of both streamline directions, one pair per step, reduced 32 at a
// time: step 2^n merges with the step before it at distance 16 >> n, so 16 steps (32 sums) take 31
// exchanges and leave each lane with one finished sum, which it adds to its tap; a butterfly per step
// takes five shuffles and a 64-bit shared atomic for every pair.  Every lane of the warp calls.
struct TapSums {
  float h1, h2, h3, h4;  // waiting for their partner at each level
  __device__ __forceinline__ void step(int i, float vb, float vf, int lb, int lf, long long* s_taps) {  // i = 1, 2, ...
    const int n = i - 1;
    float x = exchange(vb, vf, 16);
    if (!(n & 1)) {
      h1 = x;
      return;
    }
    x = exchange(h1, x, 8);
    if (!(n & 2)) {
      h2 = x;
      return;
    }
    x = exchange(h2, x, 4);
    if (!(n & 4)) {
      h3 = x;
      return;
    }
    x = exchange(h3, x, 2);
    if (!(n & 8)) {
      h4 = x;
      return;
    }
    x = exchange(h4, x, 1);
    const int lane = threadIdx.x & 31;
    const int j = (n & ~15) + 1 + (((lane >> 3) & 1) | ((lane >> 1) & 2) | ((lane << 1) & 4) | ((lane << 3) & 8));
    if (lane & 16) {
      if (j <= lf) fixed_add(s_taps + lb + j, x);
    } else if (j <= lb) {
      fixed_add(s_taps + lb - j, x);
    }
  }
  // the steps after the last one, up to a whole block of 16
  __device__ __forceinline__ void finish(int i, int lb, int lf, long long* s_taps) {
    for (; (i - 1) & 15; ++i) step(i, 0.0f, 0.0f, lb, lf, s_taps);
  }
};

// 1D LINEAR + CLAMP_TO_EDGE lookup decomposed: entries i0, i1, weight t of i1, and whether the
// coordinate lies strictly inside the interpolation range (derivative in s = 256 there, else 0).
struct Lut {
  int i0, i1;
  float t;
  bool inside;
};
__device__ __forceinline__ Lut lut(float s) {
  Lut L;
  float u = fmaf(s, (float)VVLIC_TF_ENTRIES, -0.5f);
  L.inside = u >= 0.0f && u < (float)(VVLIC_TF_ENTRIES - 1);
  u = fminf(fmaxf(u, -1.0f), (float)VVLIC_TF_ENTRIES);
  const float fl = floorf(u);
  L.t = u - fl;
  const int b = (int)fl;
  L.i0 = min(max(b, 0), VVLIC_TF_ENTRIES - 1);
  L.i1 = min(max(b + 1, 0), VVLIC_TF_ENTRIES - 1);
  return L;
}

// Unlit source of one sample from its tape record (illumLIC, inc_illum.glsl:158-172).
struct Src {
  Lut lt, lo;
  float4 tf;
  float op, base, alpha;
  float3 col;
};
__device__ __forceinline__ Src unlit_source(const RenderArgs& a, const float* s_tf, float I, float tfc) {
  Src r;
  r.lt = lut(tfc);
  const float4 t0 = reinterpret_cast<const float4*>(s_tf)[r.lt.i0], t1 = reinterpret_cast<const float4*>(s_tf)[r.lt.i1];
  r.tf = lerp4(t0, t1, r.lt.t);
  r.lo = lut(I * 1.3f);
  const float* op = s_tf + 4 * VVLIC_TF_ENTRIES;
  r.op = lerpf(op[r.lo.i0], op[r.lo.i1], r.lo.t);
  const float a0 = r.op * r.tf.w;
  r.base = 1.0f - a0;
  r.alpha = 1.0f - powf(fmaxf(r.base, 0.0f), a.alpha_corr);
  r.col = f3(I * r.tf.x * a.illum_scale, I * r.tf.y * a.illum_scale, I * r.tf.z * a.illum_scale);
  return r;
}
__device__ __forceinline__ float4 premultiplied(const Src& s) {
  return make_float4(s.col.x * s.alpha, s.col.y * s.alpha, s.col.z * s.alpha, s.alpha);
}
// illumGradient (inc_illum.glsl:1-41) intermediates: N = n(-G), R = n(2 (L.N) N - L),
// df = sat(L.N) * illumScale, spf = sat(R.V)^e.
struct LitT {
  float3 L, V, N, Rv;
  float mlen, rlen, ln, rv, df, spf;
};
__device__ __forceinline__ LitT lit_setup(const RenderArgs& a, float3 G, float3 pos, float3 dir) {
  LitT t;
  t.L = light_dir(a, pos);
  t.V = norm3(scl3(dir, -1.0f));
  const float3 m = f3(-G.x, -G.y, -G.z);
  t.mlen = sqrtf(dot3(m, m));
  t.N = norm3(m);
  t.ln = dot3(t.L, t.N);
  const float3 r = sub3(scl3(t.N, 2.0f * t.ln), t.L);
  t.rlen = sqrtf(dot3(r, r));
  t.Rv = norm3(r);
  t.rv = dot3(t.Rv, t.V);
  t.spf = powf(__saturatef(t.rv), a.spec_exp);
  t.df = __saturatef(t.ln) * a.illum_scale;
  return t;
}
__device__ __forceinline__ float3 lit_color(const RenderArgs& a, const LitT& t, float4 tf, float I) {
  return f3((tf.x * I * (a.light_diff[0] * t.df + 0.3f + a.light_amb[0]) + a.light_spec[0] * t.spf * I) * a.illum_scale,
            (tf.y * I * (a.light_diff[1] * t.df + 0.3f + a.light_amb[1]) + a.light_spec[1] * t.spf * I) * a.illum_scale,
            (tf.z * I * (a.light_diff[2] * t.df + 0.3f + a.light_amb[2]) + a.light_spec[2] * t.spf * I) * a.illum_scale);
}
// Reverse mode of lit_color for a colour cotangent dcol: dL/dtf.rgb, dL/dI, dL/dG.  sat() has
// derivative 1 strictly inside (0, 1).
__device__ __forceinline__ void lit_vjp(const RenderArgs& a, const LitT& t, float4 tf, float I, float3 dcol,
                                        float dtf[3], float* dI, float3* dG) {
  const float is = a.illum_scale;
  const float d[3] = {dcol.x, dcol.y, dcol.z}, tfc[3] = {tf.x, tf.y, tf.z};
  float cdf = 0.0f, cspf = 0.0f, di = 0.0f;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) {
    const float k = a.light_diff[ch] * t.df + 0.3f + a.light_amb[ch];
    dtf[ch] = d[ch] * I * k * is;
    di += d[ch] * (tfc[ch] * k + a.light_spec[ch] * t.spf) * is;
    cdf += d[ch] * tfc[ch] * I * a.light_diff[ch] * is;
    cspf += d[ch] * a.light_spec[ch] * I * is;
  }
  *dI = di;
  float3 gN = f3(0.f, 0.f, 0.f);
  if (t.ln > 0.0f && t.ln < 1.0f) gN = scl3(t.L, cdf * is);
  if (t.rv > 0.0f && t.rv < 1.0f && t.rlen > 0.0f && cspf != 0.0f) {
    const float dspf = cspf * a.spec_exp * powf(t.rv, a.spec_exp - 1.0f);
    const float3 gR = scl3(t.V, dspf);
    const float3 gr = scl3(sub3(gR, scl3(t.Rv, dot3(t.Rv, gR))), 1.0f / t.rlen);
    gN = add3(gN, add3(scl3(t.L, 2.0f * dot3(t.N, gr)), scl3(gr, 2.0f * t.ln)));
  }
  *dG = t.mlen > 0.0f ? scl3(sub3(gN, scl3(t.N, dot3(t.N, gN))), -1.0f / t.mlen) : f3(0.f, 0.f, 0.f);
}
__device__ __forceinline__ float3 tape_gradient(const RenderArgs& a, size_t idx) {
  const uint2 v = a.tape_g[idx];
  const float2 xy = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
  const float2 z0 = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
  return f3(xy.x, xy.y, z0.x);
}

// gI * n + gG . g of a tap
template <bool GRAD> __device__ __forceinline__ float tap_dot(float4 n, float gI, float3 gG) {
  return GRAD ? fmaf(gI, n.w, gG.x * n.x + gG.y * n.y + gG.z * n.z) : gI * n.w;
}

// Walk the streamlines of the LIC at `pos` once more and add gI * n_j (+ gG . g_j with noise
// gradients) to the tap accumulators.  Every lane of the warp takes part in each reduction;
// lanes with zero cotangents skip the fetches.
template <int ST, int FL, int NL, int INTEG, bool GRAD>
__device__ __forceinline__ void tap_gradients(const RenderArgs& a, float3 pos, float gI, float3 gG, long long* s_taps) {
  const bool act = gI != 0.0f || (GRAD && (gG.x != 0.0f || gG.y != 0.0f || gG.z != 0.0f));
  const int lb = a.lb, lf = a.lf, both = min(lb, lf), L = max(lb, lf);
  float4 f0 = make_float4(0.f, 0.f, 0.f, 0.f);
  float v0 = 0.0f;
  if (act) {
    f0 = Field<ST, FL>::sample(a, pos);
    v0 = tap_dot<GRAD>(noise_tap<NL, GRAD>(a, pos), gI, gG);
  }
  warp_fixed_add(s_taps + lb, v0);
  float3 pb = pos, pf = pos;
  float4 sb = f0, sf = f0;
  TapSums sums;
  int i = 1;
  for (; i <= both; ++i) {
    float vb = 0.0f, vf = 0.0f;
    if (act) {
      float2 n[4];
      pb = lic_step<ST, FL, INTEG>(a, pb, sb, -1.0f);
      pf = lic_step<ST, FL, INTEG>(a, pf, sf, 1.0f);
      noise_tap2<NL, GRAD>(a, pb, pf, n);
      vb = GRAD ? tap_dot<true>(make_float4(n[0].x, n[1].x, n[2].x, n[3].x), gI, gG) : gI * n[3].x;
      vf = GRAD ? tap_dot<true>(make_float4(n[0].y, n[1].y, n[2].y, n[3].y), gI, gG) : gI * n[3].y;
    }
    sums.step(i, vb, vf, lb, lf, s_taps);
  }
  for (; i <= L; ++i) {
    float vb = 0.0f, vf = 0.0f;
    if (act) {
      if (i <= lb) {
        pb = lic_step<ST, FL, INTEG>(a, pb, sb, -1.0f);
        vb = tap_dot<GRAD>(noise_tap<NL, GRAD>(a, pb), gI, gG);
      } else {
        pf = lic_step<ST, FL, INTEG>(a, pf, sf, 1.0f);
        vf = tap_dot<GRAD>(noise_tap<NL, GRAD>(a, pf), gI, gG);
      }
    }
    sums.step(i, vb, vf, lb, lf, s_taps);
  }
  sums.finish(i, lb, lf, s_taps);
}

// tap_gradients of two samples of each lane's ray: four independent streamline chains per thread, and per tap the
// two samples' contributions are added in the lane before the warp sum.  A lane walks both samples' streamlines
// when either has a non-zero cotangent; the other's terms are then zero.
template <int ST, int FL, int NL, int INTEG, bool GRAD>
__device__ __forceinline__ void tap_gradients2(const RenderArgs& a, float3 pa, float gIa, float3 gGa, float3 pc, float gIc,
                                               float3 gGc, long long* s_taps) {
  const bool act = gIa != 0.0f || gIc != 0.0f ||
                   (GRAD && (gGa.x != 0.0f || gGa.y != 0.0f || gGa.z != 0.0f || gGc.x != 0.0f || gGc.y != 0.0f ||
                             gGc.z != 0.0f));
  const int lb = a.lb, lf = a.lf, L = max(lb, lf);
  float4 fa = make_float4(0.f, 0.f, 0.f, 0.f), fc = fa;
  float v0 = 0.0f;
  const auto dot2 = [&](const float2 (&n)[4], bool second, float gI, float3 gG) {
    return second ? (GRAD ? tap_dot<true>(make_float4(n[0].y, n[1].y, n[2].y, n[3].y), gI, gG) : gI * n[3].y)
                  : (GRAD ? tap_dot<true>(make_float4(n[0].x, n[1].x, n[2].x, n[3].x), gI, gG) : gI * n[3].x);
  };
  if (act) {
    fa = Field<ST, FL>::sample(a, pa);
    fc = Field<ST, FL>::sample(a, pc);
    float2 n[4];
    noise_tap2<NL, GRAD>(a, pa, pc, n);
    v0 = dot2(n, false, gIa, gGa) + dot2(n, true, gIc, gGc);
  }
  warp_fixed_add(s_taps + lb, v0);
  float3 p0 = pa, p1 = pa, p2 = pc, p3 = pc;
  float4 s0 = fa, s1 = fa, s2 = fc, s3 = fc;
  TapSums sums;
  int i = 1;
  for (; i <= L; ++i) {
    float vb = 0.0f, vf = 0.0f;
    if (act) {
      float2 n[4];
      if (i <= lb) {
        p0 = lic_step<ST, FL, INTEG>(a, p0, s0, -1.0f);
        p2 = lic_step<ST, FL, INTEG>(a, p2, s2, -1.0f);
      }
      if (i <= lf) {
        p1 = lic_step<ST, FL, INTEG>(a, p1, s1, 1.0f);
        p3 = lic_step<ST, FL, INTEG>(a, p3, s3, 1.0f);
      }
      if (i <= lb) {
        noise_tap2<NL, GRAD>(a, p0, p2, n);
        vb = dot2(n, false, gIa, gGa) + dot2(n, true, gIc, gGc);
      }
      if (i <= lf) {
        noise_tap2<NL, GRAD>(a, p1, p3, n);
        vf = dot2(n, false, gIa, gGa) + dot2(n, true, gIc, gGc);
      }
    }
    sums.step(i, vb, vf, lb, lf, s_taps);
  }
  sums.finish(i, lb, lf, s_taps);
}

// A sample's source recomputed from its tape record: what the blend, the lookups and the shading
// need again in the reverse step.
template <bool GRAD> struct Sample {
  Src s;
  LitT lt;       // GRAD
  float3 ld;     // line lighting: colour = tf.rgb * I * ld + ...
  float I;
};
template <int ST, int FL, bool GRAD>
__device__ __forceinline__ Sample<GRAD> tape_sample(const RenderArgs& a, const float* s_tf, bool line, size_t idx,
                                                    float3 pos, float3 dir) {
  Sample<GRAD> q;
  const float2 rec = a.tape_is[idx];
  q.I = rec.x;
  q.s = unlit_source(a, s_tf, rec.x, rec.y);
  if (GRAD) {
    q.lt = lit_setup(a, tape_gradient(a, idx), pos, dir);
    q.s.col = lit_color(a, q.lt, q.s.tf, q.I);
  } else if (line) {  // (ld and the specular part are independent of TF, taps and I)
    float3 sf;
    line_factors(a, pos, dir, Field<ST, FL>::sample(a, pos), q.ld, sf);
    q.s.col = f3(q.s.tf.x * q.I * q.ld.x + sf.x, q.s.tf.y * q.I * q.ld.y + sf.y, q.s.tf.z * q.I * q.ld.z + sf.z);
  }
  return q;
}
// The source as blend() takes it (colour not yet multiplied by alpha), matching shade().
__device__ __forceinline__ float4 source_rgba(const Src& s) { return make_float4(s.col.x, s.col.y, s.col.z, s.alpha); }

// The image cotangent g through clamp((1 - Dp.a) * sv + Dp) (derivative 1 on [0, 1]) to the
// one before the sample; ds: the cotangent of the premultiplied source.
__device__ __forceinline__ float4 blend_vjp(float4 g, float4 sv, float4 Dp, float4& ds) {
  const float om = 1.0f - Dp.w;
  const float ux = fmaf(om, sv.x, Dp.x), uy = fmaf(om, sv.y, Dp.y), uz = fmaf(om, sv.z, Dp.z), uw = fmaf(om, sv.w, Dp.w);
  const float gx = (ux >= 0.f && ux <= 1.f) ? g.x : 0.f, gy = (uy >= 0.f && uy <= 1.f) ? g.y : 0.f,
              gz = (uz >= 0.f && uz <= 1.f) ? g.z : 0.f, gw = (uw >= 0.f && uw <= 1.f) ? g.w : 0.f;
  ds = make_float4(om * gx, om * gy, om * gz, om * gw);
  float4 gp = make_float4(gx, gy, gz, gw);
  gp.w -= gx * sv.x + gy * sv.y + gz * sv.z + gw * sv.w;
  return gp;
}

// Reverse step of one sample from the cotangent ds of its premultiplied source: alpha correction,
// opacity and TF lookups and the shading.  Adds the TF and opacity cotangents to the block
// accumulators and returns those of the LIC intensity (gI, scaled by the intensity scale) and of
// the gradient sum (gG).
template <bool GRAD>
__device__ __forceinline__ void sample_cotangent(const RenderArgs& a, const float* s_tf, bool line,
                                                 const Sample<GRAD>& q, float4 ds, long long* s_acc, float& gI,
                                                 float3& gG) {
  const Src& s = q.s;
  // s = (col * alpha, alpha)
  const float dcx = ds.x * s.alpha, dcy = ds.y * s.alpha, dcz = ds.z * s.alpha;
  const float dalpha = ds.x * s.col.x + ds.y * s.col.y + ds.z * s.col.z + ds.w;
  const float dba = s.base > 0.0f ? a.alpha_corr * powf(s.base, a.alpha_corr - 1.0f) : 0.0f;
  const float da0 = dalpha * dba;
  // a0 = opacity(1.3 I) * tf.a
  const float dop = da0 * s.tf.w, dtfa = da0 * s.op;
  fixed_add(s_acc + kAccOpac + s.lo.i0, dop * (1.0f - s.lo.t));
  fixed_add(s_acc + kAccOpac + s.lo.i1, dop * s.lo.t);
  const float* op = s_tf + 4 * VVLIC_TF_ENTRIES;
  float dI = s.lo.inside ? dop * (op[s.lo.i1] - op[s.lo.i0]) * (float)VVLIC_TF_ENTRIES * 1.3f : 0.0f;
  float dtf[4];
  dtf[3] = dtfa;
  if (GRAD) {
    float dIc;
    lit_vjp(a, q.lt, s.tf, q.I, f3(dcx, dcy, dcz), dtf, &dIc, &gG);
    dI += dIc;
  } else if (line) {
    dtf[0] = dcx * q.I * q.ld.x;
    dtf[1] = dcy * q.I * q.ld.y;
    dtf[2] = dcz * q.I * q.ld.z;
    dI += dcx * s.tf.x * q.ld.x + dcy * s.tf.y * q.ld.y + dcz * s.tf.z * q.ld.z;
  } else {  // col = I * tf.rgb * illumScale
    const float ci = q.I * a.illum_scale;
    dtf[0] = dcx * ci;
    dtf[1] = dcy * ci;
    dtf[2] = dcz * ci;
    dI += (dcx * s.tf.x + dcy * s.tf.y + dcz * s.tf.z) * a.illum_scale;
  }
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    fixed_add(s_acc + kAccTF + 4 * s.lt.i0 + ch, dtf[ch] * (1.0f - s.lt.t));
    fixed_add(s_acc + kAccTF + 4 * s.lt.i1 + ch, dtf[ch] * s.lt.t);
  }
  gI = dI * a.intensity_scale;
}

template <int ST, int FL, int NL, int INTEG, bool GRAD>
__global__ void __launch_bounds__(kThreads, VVLIC_ADJ_MIN_BLOCKS)
    adjoint_kernel(const __grid_constant__ RenderArgs a, const float4* __restrict__ g_img, long long* acc, unsigned ntiles,
                   unsigned* __restrict__ next) {
  __shared__ __align__(16) float s_tf[5 * VVLIC_TF_ENTRIES];
  __shared__ long long s_acc[kAccSize];
  for (int i = threadIdx.x; i < kAccSize; i += blockDim.x) s_acc[i] = 0;
  load_tf(a, s_tf);  // includes __syncthreads
  constexpr int S = 8, R = 32 / S;
  const int lane = threadIdx.x & 31, k = lane / R, r = lane % R;
  const unsigned tiles_x = (a.W + 1) / 2;
  const bool line = !GRAD && (a.illum == VVLIC_ILLUM_ZOECKLER || a.illum == VVLIC_ILLUM_MALLO);
  for (;;) {
    unsigned t = 0;
    if (lane == 0) t = atomicAdd(next, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= ntiles) break;
    unsigned tx = t % tiles_x, ty = t / tiles_x;
    if (GRAD && INTEG == VVLIC_RK4) {
      // up strips of 64 pixels, so that the rays in flight are a block of the image: one 600^2 lit RK4
      // view of 320^3, forward and adjoint, 194.9 -> 170.5 ms, 1024^2 of 512^3 930 -> 891 (unlit +0.3 %)
      constexpr unsigned strip = 32;
      const unsigned tiles_y = (a.H + 1) / 2;
      const unsigned col = t / (strip * tiles_y) * strip, rest = t - col * tiles_y, width = min(strip, tiles_x - col);
      tx = col + rest % width;
      ty = rest / width;
    }
    const int px = (int)tx * 2 + (r & 1), py = (int)ty * 2 + (r >> 1);
    float3 pos0 = f3(0.f, 0.f, 0.f), dir = f3(0.f, 0.f, 0.f);
    int n = 0;  // samples of this lane's ray
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (px < a.W && py < a.H && ray_setup(a, px, py, pos0, dir)) {
      const size_t ray = (size_t)py * a.W + px;
      n = (int)min(a.tape_n[ray], (uint32_t)a.tape_stride);
      g = g_img[ray];
    }
    const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
    for (int seg = (most + kSegment - 1) / kSegment - 1; seg >= 0; --seg) {
      const int cnt = min(max(n - seg * kSegment, 0), kSegment), top = min(most - seg * kSegment, kSegment);
      float4 D = make_float4(0.f, 0.f, 0.f, 0.f);
      float3 p0 = f3(0.f, 0.f, 0.f);
      if (cnt > 0) {
        size_t ce = tape_ck_entry(a, px, py, seg);
        if (!in_range(a, (long long)ce + 32, tape_ck_entries(a), VVLIC_CHECK_TAPE)) ce = 0;
        const float4 p4 = a.tape_ck[ce];
        p0 = f3(p4.x, p4.y, p4.z);
        D = a.tape_ck[ce + 32];
      }
      for (int j = 0; j < k; ++j) p0 = march(p0, dir, a.step_size);  // of this lane's sample in chunk 0
      // (The loops over a chunk stay rolled: unrolled, the kernel ran out of instruction cache, 1.2 of the
      // 10 stall cycles per issue, and the fit step took 38.5 ms instead of 37.3.)
      // compositing state at the start of each chunk: chunk c's in the lanes of sample c
      const int last = (top + S - 1) / S - 1;
      float4 Dstart = D;
      float3 p = p0;
      for (int c = 0; c < last; ++c) {
        float4 src = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c * S + k < cnt)
          src = source_rgba(
              tape_sample<ST, FL, GRAD>(a, s_tf, line, tape_entry_checked(a, px, py, seg * kSegment + c * S + k), p, dir).s);
#pragma unroll 1
        for (int j = 0; j < S; ++j) {
          const float4 s = shfl4(src, j * R + r);
          if (c * S + j < cnt) D = blend(D, s);
        }
        if (k == c + 1) Dstart = D;
        for (int j = 0; j < S; ++j) p = march(p, dir, a.step_size);
      }
      for (int c = last; c >= 0; --c) {
        p = p0;
        for (int j = 0; j < c * S; ++j) p = march(p, dir, a.step_size);
        const bool valid = c * S + k < cnt;
        Sample<GRAD> q;
        float4 src = make_float4(0.f, 0.f, 0.f, 0.f), sv = src;
        if (valid) {
          q = tape_sample<ST, FL, GRAD>(a, s_tf, line, tape_entry_checked(a, px, py, seg * kSegment + c * S + k), p, dir);
          src = source_rgba(q.s);
          sv = premultiplied(q.s);
        }
        // state before each sample; this lane keeps its own sample's
        float4 Dmine = shfl4(Dstart, c * R + r);
        D = Dmine;
#pragma unroll 1
        for (int j = 0; j < S; ++j) {
          const float4 s = shfl4(src, j * R + r);
          if (j == k) Dmine = D;
          if (c * S + j < cnt) D = blend(D, s);
        }
        float4 ds = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int j = S - 1; j >= 0; --j) {
          const float4 svj = shfl4(sv, j * R + r), Dj = shfl4(Dmine, j * R + r);
          if (c * S + j < cnt) {
            float4 dsj;
            g = blend_vjp(g, svj, Dj, dsj);
            if (j == k) ds = dsj;
          }
        }
        float gI = 0.0f;
        float3 gG = f3(0.f, 0.f, 0.f);
        if (valid) sample_cotangent<GRAD>(a, s_tf, line, q, ds, s_acc, gI, gG);
        const bool need = gI != 0.0f || (GRAD && (gG.x != 0.0f || gG.y != 0.0f || gG.z != 0.0f));
        if (__any_sync(0xffffffffu, need)) tap_gradients<ST, FL, NL, INTEG, GRAD>(a, p, gI, gG, s_acc + kAccTaps);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kAccSize; i += blockDim.x)
    if (s_acc[i] != 0) atomicAdd(reinterpret_cast<unsigned long long*>(acc + i), (unsigned long long)s_acc[i]);
}

// The same by a lane per ray on 8x4-pixel tiles: a segment's positions and states in a local array, its samples
// last to first, in RK4 two at a time.  Lit RK4 with up to 96 registers (5 CTAs): 2048^2 view along an axis of a
// 512^3 field, L = 60, 1274 ms against 1339 with 80 and 1333 with 128.
template <int INTEG, bool GRAD> constexpr int ray_min_blocks() {
  return GRAD && INTEG == VVLIC_RK4 ? VVLIC_ADJ_MIN_BLOCKS - 1 : VVLIC_ADJ_MIN_BLOCKS;
}
template <int ST, int FL, int NL, int INTEG, bool GRAD>
__global__ void __launch_bounds__(kThreads, ray_min_blocks<INTEG, GRAD>())
    adjoint_ray_kernel(const __grid_constant__ RenderArgs a, const float4* __restrict__ g_img, long long* acc,
                       unsigned ntiles, unsigned* __restrict__ next) {
  __shared__ __align__(16) float s_tf[5 * VVLIC_TF_ENTRIES];
  __shared__ long long s_acc[kAccSize];
  for (int i = threadIdx.x; i < kAccSize; i += blockDim.x) s_acc[i] = 0;
  load_tf(a, s_tf);  // includes __syncthreads
  constexpr int P = INTEG == VVLIC_RK4 ? 2 : 1;
  const int lane = threadIdx.x & 31;
  const unsigned tiles_x = (a.W + 7) / 8, tiles_y = (a.H + 3) / 4;
  const bool line = !GRAD && (a.illum == VVLIC_ILLUM_ZOECKLER || a.illum == VVLIC_ILLUM_MALLO);
  float4 Dloc[kSegment];
  float3 Ploc[kSegment];
  for (;;) {
    unsigned t = 0;
    if (lane == 0) t = atomicAdd(next, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= ntiles) break;
    constexpr unsigned strip = 8;  // up strips of 64 pixels
    const unsigned col = t / (strip * tiles_y) * strip, rest = t - col * tiles_y, width = min(strip, tiles_x - col);
    const int x0 = (int)(col + rest % width) * 8, y0 = (int)(rest / width) * 4;
    const int px = x0 + (lane & 7), py = y0 + (lane >> 3);
    float3 pos0 = f3(0.f, 0.f, 0.f), dir = f3(0.f, 0.f, 0.f);
    int n = 0;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (px < a.W && py < a.H && ray_setup(a, px, py, pos0, dir)) {
      const size_t ray = (size_t)py * a.W + px;
      n = (int)min(a.tape_n[ray], (uint32_t)a.tape_stride);
      g = g_img[ray];
    }
    const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
    for (int seg = (longest + kSegment - 1) / kSegment - 1; seg >= 0; --seg) {
      const int cnt = min(max(n - seg * kSegment, 0), kSegment), top = min(longest - seg * kSegment, kSegment);
      if (cnt > 0) {
        size_t ce = tape_ck_entry(a, px, py, seg);
        if (!in_range(a, (long long)ce + 32, tape_ck_entries(a), VVLIC_CHECK_TAPE)) ce = 0;
        const float4 p4 = a.tape_ck[ce];
        float3 p = f3(p4.x, p4.y, p4.z);
        float4 D = a.tape_ck[ce + 32];
        for (int j = 0; j < cnt; ++j) {
          Ploc[j] = p;
          Dloc[j] = D;
          D = blend(D, source_rgba(tape_sample<ST, FL, GRAD>(a, s_tf, line, tape_entry_checked(a, px, py, seg * kSegment + j),
                                                             p, dir).s));
          p = march(p, dir, a.step_size);
        }
      }
      // the cotangents of sample j: of its intensity (gI) and gradient sum (gG)
      const auto back = [&](int j, float& gI, float3& gG, float3& pk) {
        gI = 0.0f;
        gG = f3(0.f, 0.f, 0.f);
        pk = f3(0.f, 0.f, 0.f);
        if (j < 0 || j >= cnt) return false;
        pk = Ploc[j];
        const Sample<GRAD> q =
            tape_sample<ST, FL, GRAD>(a, s_tf, line, tape_entry_checked(a, px, py, seg * kSegment + j), pk, dir);
        float4 ds;
        g = blend_vjp(g, premultiplied(q.s), Dloc[j], ds);
        sample_cotangent<GRAD>(a, s_tf, line, q, ds, s_acc, gI, gG);
        return gI != 0.0f || (GRAD && (gG.x != 0.0f || gG.y != 0.0f || gG.z != 0.0f));
      };
      for (int j = (top + P - 1) / P * P - 1; j >= 0; j -= P) {
        float gI, gI1;
        float3 gG, gG1, p, p1;
        bool need = back(j, gI, gG, p);
        if constexpr (P == 2) {
          need |= back(j - 1, gI1, gG1, p1);
          if (__any_sync(0xffffffffu, need))
            tap_gradients2<ST, FL, NL, INTEG, GRAD>(a, p, gI, gG, p1, gI1, gG1, s_acc + kAccTaps);
        } else {
          if (__any_sync(0xffffffffu, need)) tap_gradients<ST, FL, NL, INTEG, GRAD>(a, p, gI, gG, s_acc + kAccTaps);
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kAccSize; i += blockDim.x)
    if (s_acc[i] != 0) atomicAdd(reinterpret_cast<unsigned long long*>(acc + i), (unsigned long long)s_acc[i]);
}

// A lane per ray where groups of eight samples lose:
//   frames of short rays (head_samples), 512 x 512 x 4 volume, 1024^2, groups / lane per ray: unlit 0.40 / 0.17 ms,
//     lit 2.35 / 1.27, RK4 2.76 / 2.13; 300^2 0.07 / 0.06, 0.25 / 0.19, 0.30 / 0.27;
//   frames whose rays may end early, from 16 times as many 2x2-ray tiles as resident warps (RK4: 64): all
//     opaque, 1024^2, 0.31 / 0.06, 0.44 / 0.09, 0.45 / 0.11 ms; rays that go on 5.3 / 3.3, 33.0 / 24.7, 39.5 / 41.5, but at
//     450^2 1.1 / 1.4, 6.8 / 6.9, 8.5 / 11.0;
//   the largest lit RK4 frames, from 192 times as many, or 64 where rows of pixels lie along rows of texels: views of
//     a 512^3 field so / turned, L = 60, 2048^2 1456 / 1274 and 1494 / 1470 ms (before the groups 1312 and 1491),
//     1024^2 420 / 400 and 480 / 517 (387 and 512);
//   large frames of the other kinds, the sooner the shorter the streamlines: all eight lanes of a ray blend its
//     samples, so the compositing costs the groups more.  128^3, L = 30, default / random TF: lit Heun 500^2 5.0 / 5.1 and 8.0 / 7.8, 650^2 8.2 / 6.9
//     and 13.2 / 11.8, 1100^2 23.0 / 15.8 and 37.1 / 29.9; unlit 650^2 1.34 / 0.76 and 3.74 / 4.93, 800^2 2.00 / 1.08 and 5.49 / 6.19;
//     unlit RK4 1100^2 3.78 / 2.10 and 13.7 / 15.6.  192^3, L = 60: lit Heun 500^2 15.9 / 16.3 and 20.3 / 22.4, 650^2 26.3 / 25.6 and
//     33.7 / 33.3; unlit 800^2 3.2 / 2.8 and 12.5 / 16.7, 1100^2 6.0 / 4.1 and 22.8 / 25.1; unlit RK4 1100^2 6.1 / 5.4 and 34.8 / 41.9.
//     96^3, L = 10: lit Heun 500^2 1.56 / 0.94 and 3.43 / 2.81; RK4 800^2 unlit 1.56 / 0.89 and 3.45 / 3.53, lit 3.88 / 2.94 and
//     9.82 / 9.77.
template <int INTEG, bool GRAD> static bool lane_per_ray(const RenderArgs& a, int num_sms) {
  const long long tiles = cast_tiles(a), resident = resident_warps(num_sms);
  if (head_samples(a, num_sms) == 0xffffffffu) return true;
  if (may_end(a) && tiles >= (INTEG == VVLIC_RK4 && a.end_share < 0.5f ? 64 : 16) * resident) return true;
  const int L = std::max(a.lb, a.lf);
  int line = 0;
  if (INTEG != VVLIC_RK4) line = GRAD ? (L <= 24 ? 16 : 24) : (L <= 36 ? 40 : 64);
  else if (GRAD) line = L <= 24 ? 40 : (a.along_rows ? 64 : 192);
  else line = L <= 24 ? 40 : (L <= 36 ? 64 : 128);
  return tiles >= line * resident;
}

template <typename Kernel>
static cudaError_t launch_tiles(Kernel kern, const RenderArgs& a, const float4* g_img, long long* acc, unsigned ntiles,
                                unsigned* next, int num_sms, cudaStream_t s) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, 0);
  if (e != cudaSuccess) return e;
  const int grid = (int)std::min<unsigned>((ntiles + kWarps - 1) / kWarps, (unsigned)(std::max(1, per_sm) * num_sms));
  kern<<<grid, kThreads, 0, s>>>(a, g_img, acc, ntiles, next);
  return cudaGetLastError();
}

template <int ST, int FL, int NL, int INTEG, bool GRAD>
static cudaError_t launch_adjoint_one(const RenderArgs& a, const float4* g_img, long long* acc, unsigned* next,
                                      int num_sms, cudaStream_t s) {
  const auto tiles = [&](int w, int h) { return (unsigned)((a.W + w - 1) / w) * (unsigned)((a.H + h - 1) / h); };
  if (lane_per_ray<INTEG, GRAD>(a, num_sms))
    return launch_tiles(adjoint_ray_kernel<ST, FL, NL, INTEG, GRAD>, a, g_img, acc, tiles(8, 4), next, num_sms, s);
  return launch_tiles(adjoint_kernel<ST, FL, NL, INTEG, GRAD>, a, g_img, acc, tiles(2, 2), next, num_sms, s);
}

template <int ST, int FL, int NL, bool GRAD>
static cudaError_t launch_adjoint_integ(const RenderArgs& a, int integ, const float4* g_img, long long* acc,
                                        unsigned* next, int num_sms, cudaStream_t s) {
  if (integ == VVLIC_EULER) return launch_adjoint_one<ST, FL, NL, VVLIC_EULER, GRAD>(a, g_img, acc, next, num_sms, s);
  if (integ == VVLIC_HEUN) return launch_adjoint_one<ST, FL, NL, VVLIC_HEUN, GRAD>(a, g_img, acc, next, num_sms, s);
  return launch_adjoint_one<ST, FL, NL, VVLIC_RK4, GRAD>(a, g_img, acc, next, num_sms, s);
}

template <int ST, int FL, int NL>
static cudaError_t launch_adjoint_layout(const RenderArgs& a, int integ, bool lit, const float4* g_img,
                                         long long* acc, unsigned* next, int num_sms, cudaStream_t s) {
  return lit ? launch_adjoint_integ<ST, FL, NL, true>(a, integ, g_img, acc, next, num_sms, s)
             : launch_adjoint_integ<ST, FL, NL, false>(a, integ, g_img, acc, next, num_sms, s);
}

template <int ST>
static cudaError_t launch_adjoint_storage(const RenderArgs& a, int sampler, int integ, bool lit, const float4* g_img,
                                          long long* acc, unsigned* next, int num_sms, cudaStream_t s) {
  switch (sampler) {
    case VVLIC_SAMPLER_GATHER: return launch_adjoint_layout<ST, kGather, kGather>(a, integ, lit, g_img, acc, next, num_sms, s);
    case VVLIC_SAMPLER_CELL: return launch_adjoint_layout<ST, kCell, kCell>(a, integ, lit, g_img, acc, next, num_sms, s);
    case VVLIC_SAMPLER_TEXTURE:
      if constexpr (ST == VVLIC_STORAGE_BF16) return cudaErrorNotSupported;  // runs as F16 (kernel_storage)
      else return launch_adjoint_layout<ST, kTexture, kTexture>(a, integ, lit, g_img, acc, next, num_sms, s);
    case VVLIC_SAMPLER_HYBRID:
      if constexpr (ST == VVLIC_STORAGE_BF16) return cudaErrorNotSupported;
      else return launch_adjoint_layout<ST, kTexture, kCellFast>(a, integ, lit, g_img, acc, next, num_sms, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vvlic
