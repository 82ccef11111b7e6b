// Adam::step (reference src/adam.rs:44-161) on one float4 of a parameter plane, shared by
// the stand-alone optimiser kernel and the projection backward that applies it in place.
#pragma once
#include "common.cuh"

namespace splat {

struct alignas(16) AdamArgs {
  float lr[4][4];  // per lane of planes 0..3; planes >= 4 use sh_rest
  float sh_rest;
  float b1, b2, c1, c2, eps;
  float r1, r2;  // 1 / c1 and 1 / c2, rounded
  int recip;     // c1 and c2 lie in the range that div_by asks for
};

// Correctly rounded quotients and square roots from fused multiply-adds, after P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor" (IBM J. Res.
// Dev. 34, 1990): with y = RN(1 / b) and a faithful q, q + y (a - b q) rounds to RN(a / b), as
// long as the remainder is exact. Unlike the operators they have no way out for operands out
// of range; adam_update keeps to the ranges named there.
__device__ __forceinline__ float div_steps(float a, float b, float y) {
  float q = a * y;
  q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);  // faithful
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
// RN(1 / b) for a b whose significand isn't all ones.
__device__ __forceinline__ float rcp_steps(float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  y = __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
  return __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
}
// RN(sqrt(x)): s ~ sqrt(x) and h ~ 1 / (2 sqrt(x)) refined together, then s + h (x - s s).
__device__ __forceinline__ float sqrt_steps(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  float s = x * y, h = 0.5f * y;
  const float d = __fmaf_rn(-s, h, 0.5f);
  s = __fmaf_rn(s, d, s);
  h = __fmaf_rn(h, d, h);
  return __fmaf_rn(__fmaf_rn(-s, s, x), h, s);
}

// lr m_hat / (sqrt(v_hat) + eps) by the operators, for every operand.
static __device__ __noinline__ float adam_quotient(float m, float v, float lr, float c1, float c2, float eps) {
  return lr * (m / c1) / (sqrtf(v / c2) + eps);
}

// adam.rs:44-61, in the reference's operation order (compiled without contraction) and to its
// bits: the new moments, and in q what p loses. Instructions bound this, not memory: with the
// operators an element took about 160, since zero moments (parameters without a gradient) and
// small operands send the division and the square root down their long way, lane by lane; the
// steps above need none of it in
//   v = 0 or 2^-126 <= v <= 2^60 (scaled by 2^80 where small, so that remainders are exact),
//   m = 0 or 2^-90 <= |m| <= 2^60 with 2^-90 <= |lr m_hat| <= 2^60 (so that no quotient and no
//   remainder overflows: |lr m_hat| / 1e-15 stays below 2^110),
// and where m is smaller, but the quotient below 2^-27 |p|, p stays what it is for any
// quotient of that size. False for everything else: q is then to come from adam_quotient.
__device__ __forceinline__ bool adam_moments(float p, float g, float& m, float& v, float lr, const AdamArgs& a,
                                             float& q) {
  m = a.b1 * m + (1.0f - a.b1) * g;
  v = a.b2 * v + (1.0f - a.b2) * g * g;
  const bool small = v < 0x1p-40f;
  const float root = sqrt_steps(div_steps(v * (small ? 0x1p80f : 1.0f), a.c2, a.r2)) * (small ? 0x1p-40f : 1.0f);
  const float den = (v == 0.0f ? v : root) + a.eps;
  const float num = lr * div_steps(m, a.c1, a.r1);
  q = div_steps(num, den, rcp_steps(den));
  q = m == 0.0f ? num : q;
  const float am = fabsf(m), ap = fabsf(p);
  const bool v_ok = v == 0.0f || (v >= 0x1p-126f && v <= 0x1p60f);
  const bool m_ok = m == 0.0f || (fminf(am, fabsf(num)) >= 0x1p-90f && fmaxf(am, fabsf(num)) <= 0x1p60f) ||
                    (ap >= 0x1p-60f && fabsf(q) < 0x1p-27f * ap);
  return v_ok & m_ok & ((__float_as_uint(den) & 0x7FFFFFu) != 0x7FFFFFu);
}

// One float4 of plane `plane` with the learning rate of each lane's parameter group.
__device__ __forceinline__ void adam_plane(const AdamArgs& a, int plane, float4& p, const float4& g, float4& m,
                                           float4& v) {
  const float4 lr = plane < 4 ? *reinterpret_cast<const float4*>(a.lr[plane])
                              : make_float4(a.sh_rest, a.sh_rest, a.sh_rest, a.sh_rest);
  float4 q;
  const bool ok = adam_moments(p.x, g.x, m.x, v.x, lr.x, a, q.x) & adam_moments(p.y, g.y, m.y, v.y, lr.y, a, q.y) &
                  adam_moments(p.z, g.z, m.z, v.z, lr.z, a, q.z) & adam_moments(p.w, g.w, m.w, v.w, lr.w, a, q.w);
  if (!(ok && a.recip)) {
    q.x = adam_quotient(m.x, v.x, lr.x, a.c1, a.c2, a.eps);
    q.y = adam_quotient(m.y, v.y, lr.y, a.c1, a.c2, a.eps);
    q.z = adam_quotient(m.z, v.z, lr.z, a.c1, a.c2, a.eps);
    q.w = adam_quotient(m.w, v.w, lr.w, a.c1, a.c2, a.eps);
  }
  p.x -= q.x;
  p.y -= q.y;
  p.z -= q.z;
  p.w -= q.w;
}

// Bias corrections for step `step` (after the increment) and the per-lane rates.
AdamArgs make_adam_args(uint64_t step, const splat_lr& lr);

}  // namespace splat
