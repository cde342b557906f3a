// Scalar steps of the PCG iterations in the mixed path: quotients by numbers
// known before the sums are, and the step lengths of the single-reduction form.
// Float-float on the FP32 pipe throughout, since an FP64 instruction takes 66
// cycles and its division 576, but with no larger an error than FP64 products
// and differences of float-float quotients have: against 64-bit significands, a
// quotient 2^-49.0 at most and 2^-50.6 rms (float-float division: 2^-46.8 and
// 2^-49.3), alpha of the single-reduction form 2^-46.0 and 2^-48.9 (with FP64
// between float-float divisions: 2^-45.5 and 2^-48.5; with float-float products
// and reciprocals alone: 2^-45.0 and 2^-48.0), where d is three times the
// difference it enters.  The work on a reciprocal is done while the sums travel.
#pragma once
#include "df64.cuh"

namespace mfem_gpu {

// The reciprocal of a float-float number to 2^-68: float-float, and the rest.
struct df_rcp {
  df64 r;
  float rest;
};
// 1 / v: the float-float quotient r and what 1 - v r leaves, which cancels to
// 2^-45, so that the four parts of v r are exact products summed without loss.
__device__ __forceinline__ df_rcp rcp_of(df64 v) {
  const df64 r = df64(1.f) / v;
  const df64 p = two_prod(v.hi, r.hi), c = two_prod(v.hi, r.lo), e = two_prod(v.lo, r.hi);
  const df64 b = two_sum(__fsub_rn(1.f, p.hi), -p.lo), s1 = two_sum(b.hi, -c.hi), s2 = two_sum(s1.hi, -e.hi);
  const float up = __fadd_rn(__fadd_rn(s1.lo, s2.lo), b.lo);
  const float down = __fmaf_rn(v.lo, r.lo, __fadd_rn(c.lo, e.lo));
  return df_rcp{r, __fmul_rn(__fadd_rn(s2.hi, __fsub_rn(up, down)), r.hi)};
}
// a (b + rest), rounded once: the products' errors carried along.
__device__ __forceinline__ df64 df_product(df64 a, df64 b, float rest = 0.f) {
  const df64 p = two_prod(a.hi, b.hi), c = two_prod(a.hi, b.lo), e = two_prod(a.lo, b.hi);
  const df64 s = two_sum(c.hi, e.hi), t = two_sum(s.hi, p.lo), u = two_sum(p.hi, t.hi);
  const float lo = __fadd_rn(__fadd_rn(c.lo, e.lo), __fmaf_rn(a.hi, rest, __fmul_rn(a.lo, b.lo)));
  return fast_two_sum(u.hi, __fadd_rn(u.lo, __fadd_rn(__fadd_rn(s.lo, t.lo), lo)));
}
// a - b accurate relative to the result (two TwoSums: Knuth; Hida, Li, Bailey 2001).
__device__ __forceinline__ df64 df_difference(df64 a, df64 b) {
  const df64 s = two_sum(a.hi, -b.hi), t = two_sum(a.lo, -b.lo);
  const df64 u = fast_two_sum(s.hi, __fadd_rn(s.lo, t.hi));
  return fast_two_sum(u.hi, __fadd_rn(u.lo, t.lo));
}

// num / den for a den known long before num, whose reciprocal is at hand.  A
// den near the ends of FP32's range, whose reciprocal or its low part would
// not be in it, is divided by.  FP64: the division (its kernels have their own
// form of this, quotient_by).
__device__ __forceinline__ df64 by_rcp(df64 num, df64 den, const df_rcp& rcp) {
  const float m = fabsf(den.hi);
  if (m > 1e-30f && m < 1e30f) return df_product(num, rcp.r, rcp.rest);
  return num / den;
}
__device__ __forceinline__ double by_rcp(double num, double den, double) { return num / den; }
// num / den of which only the nearest float is used (to_step), with den's
// float-float reciprocal: the product, whose error is below 2^-44, unless it
// lies so near the middle of two floats that the error could decide (Ziv 1991).
__device__ __forceinline__ df64 by_rcp_step(df64 num, df64 den, df64 rcp) {
  const float m = fabsf(den.hi);
  const df64 v = num * rcp;
  if (m > 1e-30f && m < 1e30f && __fmaf_rn(v.lo, 1.f + 0x1p-17f, v.hi) == v.hi) return v;
  return by_rcp(num, den, rcp_of(den));
}
// A step length as every thread uses it.
__device__ __forceinline__ float to_step(df64 v) { return __fadd_rn(v.hi, v.lo); }
__device__ __forceinline__ double rcp_of(double) { return 0.0; }

// Step lengths of the single-reduction iteration from (r, u), (w, u), the
// previous (r, u) and alpha and their reciprocals, which are known before the
// sums are: b = g / g_prev, a = g / (d - b g / a_prev), with one division after
// them instead of three.  Mixed path: g / a_prev beside b, not behind it.
__device__ __forceinline__ df64 cgf_alpha(df64 g, df64 d, df64 b, df64 g_by_a_prev) {
  return g / df_difference(d, df_product(b, g_by_a_prev));
}
__device__ __forceinline__ void cgf_steps(df64 g, df64 d, df64 g_prev, df64 a_prev, const df_rcp& g_rcp,
                                          const df_rcp& a_rcp, df64* a, df64* b) {
  *b = by_rcp(g, g_prev, g_rcp);
  *a = cgf_alpha(g, d, *b, by_rcp(g, a_prev, a_rcp));
}
__device__ __forceinline__ void cgf_steps(double g, double d, double g_prev, double a_prev, double, double, double* a,
                                          double* b) {
  const double bn = g / g_prev;
  *b = bn;
  *a = g / (d - bn * g / a_prev);
}
// .. and after a failed verification, where the new direction is made
// A-conjugate to the last one directly: b = -(A p, u) / (p, A p), and (p_new,
// A p_new) = d + 2 b (A p, u) + b^2 (p, A p).  Once or twice a solve at most:
// the sum in FP64.
__device__ __forceinline__ void cgf_restart_steps(df64 g, df64 d, df64 su, df64 ps, df64* a, df64* b) {
  const double bn = -(su / ps).to_double();
  *b = df64(bn);
  *a = g / df64(d.to_double() + 2.0 * bn * su.to_double() + bn * bn * ps.to_double());
}

}  // namespace mfem_gpu
