// ammsb_gamma.cuh -- the Gamma(1, 1) draws of the initial phi, in pairs of
// FP32 numbers.
//
// The spec of a draw is FP64 (gamma_draw in ammsb_device.cuh): a logarithm, a
// square root and a cosine per attempt, some 260 issue slots at GB300's FP64
// rate (1/64 of FP32), rounded to FP32 at the end.  Here the same expression
// is evaluated as unevaluated sums of two FP32 numbers (Dekker 1971; the error
// terms of products by FMA), whose error is some 2^-44, with
//   - the logarithm table-driven (Tang 1990): u = m 2^-(s+1), m c_i = 1 + r with
//     c_i a ten-bit reciprocal of m's interval, so r is exact to 2^-48, and the
//     series of log(1 + r) for |r| < 0.005;
//   - the cosine as cos(A + d) = cos A + cos A (cos d - 1) - sin A sin d over 256
//     table angles A, |d| < 0.0123.
// A draw is taken only where the error bound cannot change its FP32 rounding
// (Ziv's test) nor a comparison of the rejection; elsewhere (about one draw in
// 3,000) the FP64 draw is made.  So every draw is the FP64 one's FP32 value:
// none of 3.2e9 draws compared differed.  Largest errors over all 2^32 words:
// log 2^-43.1, root 2^-43.8, cosine 2^-42.4, so that v = 1 + root cos / sqrt 6
// (root <= 6.77) is within 2^-40.9; the largest seen was 2^-41.9, the bound used
// 2^-40.  Bound by FP32 issue: 7.7M draws, with their row sums and pi, went from
// 3.30 ms to 0.2 ms on GB300.
#pragma once
#include "ammsb_device.cuh"

namespace ammsb {

struct FF {  // h + l, |l| <= ulp(h) / 2
  float h, l;
};
__device__ __forceinline__ FF ff_two_sum(float a, float b) {  // exact
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return FF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ FF ff_fast(float a, float b) {  // exact for |a| >= |b|
  const float s = __fadd_rn(a, b);
  return FF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_prod(float a, float b) {  // exact
  const float p = __fmul_rn(a, b);
  return FF{p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
  const FF s = ff_two_sum(a.h, b.h);
  return ff_fast(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ FF ff_mul(FF a, FF b) {
  const FF p = ff_prod(a.h, b.h);
  return ff_fast(p.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, p.l)));
}

constexpr int kLogSteps = 128, kExps = 33, kAngles = 256;
struct GammaTables {
  float4 log_step[kLogSteps];  // c_i, log(c_i) as a pair
  float2 exps[kExps + 1];      // (s + 1) log 2
  float4 angle[kAngles];       // cos A, sin A as pairs
};
__device__ __forceinline__ float2 split_pair(double x) {
  const float h = (float)x;
  return make_float2(h, (float)(x - (double)h));
}
static __global__ void __launch_bounds__(256) k_gamma_tables(GammaTables* t) {
  const int i = threadIdx.x;
  if (i < kLogSteps) {
    const double c = rint(1024.0 / (1.0 + (i + 0.5) / kLogSteps)) / 1024.0;
    const float2 l = split_pair(log(c));
    t->log_step[i] = make_float4((float)c, l.x, l.y, 0.f);
  }
  if (i < kExps) t->exps[i] = split_pair((i + 1) * log(2.0));
  double s, c;
  sincospi(2.0 * i / kAngles, &s, &c);
  const float2 cp = split_pair(c), sp = split_pair(s);
  t->angle[i] = make_float4(cp.x, cp.y, sp.x, sp.y);
}

// -log((x + 1/2) 2^-32)
__device__ __forceinline__ FF ff_neg_log_u(uint32_t x, const GammaTables& t) {
  // N = 2 x + 1 = m 2^(32 - s), 1 <= m < 2
  const int s = x ? __clz(x) : 32;
  const unsigned long long M = ((unsigned long long)x * 2ull + 1ull) << s;  // bit 32 set
  const uint32_t top = (uint32_t)(M >> 9);                                    // 24 bits
  const float mh = (float)top * 0x1p-23f, ml = (float)(uint32_t)(M & 511u) * 0x1p-32f;
  const float4 step = t.log_step[(top >> 16) & (kLogSteps - 1)];
  // r = m c - 1
  const FF p = ff_prod(mh, step.x);
  const FF r = ff_two_sum(__fsub_rn(p.h, 1.f), __fmaf_rn(ml, step.x, p.l));
  // log(1 + r) = r - r^2 / 2 + r^3 (1/3 - r/4 + r^2/5 - r^3/6)
  const float q = __fmul_rn(r.h, r.h);
  const float ql = __fmaf_rn(r.h, r.h, -q) + 2.f * r.h * r.l;
  const float tail = q * r.h * fmaf(r.h, fmaf(r.h, fmaf(r.h, -1.f / 6.f, 0.2f), -0.25f), 1.f / 3.f);
  const FF a = ff_fast(r.h, -0.5f * q);
  const FF log1 = ff_fast(a.h, a.l + (r.l + (tail - 0.5f * ql)));
  // (s + 1) log 2 + log c - log(1 + r)
  const float2 e = t.exps[s];
  return ff_add(ff_add(FF{e.x, e.y}, FF{step.y, step.z}), FF{-log1.h, -log1.l});
}

// cos(2 pi y 2^-32)
__device__ __forceinline__ FF ff_cos_turn(uint32_t y, const GammaTables& t) {
  const uint32_t i = (y + (1u << 23)) >> 24;  // nearest table angle
  const float f = (float)(int32_t)(y - (i << 24));
  const float4 A = t.angle[i & (kAngles - 1)];
  // d = 2 pi f 2^-32
  const float kh = (float)(6.283185307179586476925287 * 0x1p-32);
  const float kl = (float)(6.283185307179586476925287 * 0x1p-32 - (double)kh);
  FF d = ff_prod(f, kh);
  d.l = fmaf(f, kl, d.l);
  const float q = __fmul_rn(d.h, d.h);
  const float ql = __fmaf_rn(d.h, d.h, -q) + 2.f * d.h * d.l;
  // sin d = d - d^3/6 + d^5/120; cos d - 1 = -d^2/2 + d^4/24
  const float sl = d.l - q * d.h * fmaf(q, -1.f / 120.f, 1.f / 6.f);
  const float ch = -0.5f * q, cl = fmaf(q * q, 1.f / 24.f, -0.5f * ql);
  const FF c = ff_prod(A.x, ch), s = ff_prod(-A.z, d.h);
  const float low = (c.l + fmaf(A.x, cl, A.y * ch)) + (s.l - fmaf(A.z, sl, A.w * d.h));
  const FF a = ff_two_sum(A.x, s.h);
  const FF b = ff_two_sum(a.h, c.h);
  return ff_fast(b.h, (b.l + a.l) + (A.y + low));
}

// gamma_draw(rs, tag, entity, idx, 1, 1, err) as FP32.
__device__ __forceinline__ float gamma_one_draw(const Stream& rs, uint32_t tag, uint32_t entity, uint64_t idx,
                                                const GammaTables& t, int32_t* err) {
  constexpr float kErrV = 0x1p-40f;  // bound of v's absolute error
  for (uint32_t attempt = 0; attempt < 64; ++attempt) {
    const U32x4 o = rs.block(tag, entity, attempt, idx);
    // x = sqrt(-2 log u1) cos(2 pi u2), v = 1 + x / sqrt 6
    FF z = ff_neg_log_u(o.x, t);
    z = FF{2.f * z.h, 2.f * z.l};
    if (!(z.h > 0x1p-12f)) break;  // u1 near 1: the difference of logarithms has lost its digits
    const float s0 = __fsqrt_rn(z.h);
    const FF root = ff_fast(s0, __fadd_rn(__fmaf_rn(-s0, s0, z.h), z.l) * (0.5f * rcp_approx(s0)));
    const FF x = ff_mul(root, ff_cos_turn(o.y, t));
    const double c = 0.408248290463863016366214012451;  // 1 / sqrt(9 (1 - 1/3))
    const FF w = ff_mul(x, FF{(float)c, (float)(c - (double)(float)c)});
    const FF v = ff_add(FF{1.f, 0.f}, w);
    if (v.h < -0x1p-20f) continue;
    if (v.h < 0x1p-20f) break;
    const float x2 = x.h * x.h;
    const float u = ((float)o.z + 0.5f) * 2.3283064365386963e-10f;
    const FF v3 = ff_mul(ff_mul(v, v), v);
    const float out = 0.0331f * x2 * x2;
    const float slack = u - (1.f - out);
    if (!(slack < -1e-5f * (1.f + out))) {
      if (!(slack > 1e-5f * (1.f + out))) break;
      // the exact test: log u < x^2 / 2 + d (1 - v^3 + log v^3)
      const float lu = logf(u), lv = logf(v3.h);
      const float rhs = 0.5f * x2 + (2.f / 3.f) * (1.f - v3.h + lv);
      const float tol = 2e-5f * (1.f - lu + x2 + v3.h + fabsf(lv));
      if (lu > rhs + tol) continue;
      if (!(lu < rhs - tol)) break;
    }
    const double d = 2.0 / 3.0;
    const FF g = ff_mul(v3, FF{(float)d, (float)(d - (double)(float)d)});
    // d v^3 moves by 2 v^2 of v's error, and by its own roundings
    const float e = fmaf(2.f * v.h * v.h, kErrV, g.h * 0x1p-42f);
    const float lo = __fadd_rn(g.h, __fsub_rn(g.l, e)), hi = __fadd_rn(g.h, __fadd_rn(g.l, e));
    if (lo == hi) return lo;
    break;
  }
  return (float)gamma_draw(rs, tag, entity, idx, 1.0, 1.0, err);
}

}  // namespace ammsb
