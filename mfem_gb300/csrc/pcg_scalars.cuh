// Scalar steps of the PCG iterations in the mixed path: quotients by numbers
// known before the sums are, and the step lengths of the single-reduction form.
// Float-float on the FP32 pipe throughout, since an FP64 instruction takes 66
// cycles and its division 576, but with no larger an error than FP64 products
// and differences of float-float quotients have: against 128-bit arithmetic, a
// quotient 2^-49.0 at most and 2^-50.6 rms (float-float division: 2^-46.8 and
// 2^-49.3), alpha of the single-reduction form 2^-45.9 and 2^-48.7 (with FP64
// between float-float divisions: 2^-45.7 and 2^-48.5; with float-float products
// and reciprocals alone: 2^-45.0 and 2^-48.0), where d is three times the
// difference it enters.
#pragma once
#include "df64.cuh"

namespace mfem_gpu {

// num / den with den's reciprocal (a float-float number) at hand: the product,
// corrected by its remainder.  The remainder cancels to 2^-45 of num, so the
// four parts of quotient x den are exact products summed without loss.
__device__ __forceinline__ df64 df_quotient(df64 num, df64 den, df64 rcp) {
  const df64 t = num * rcp;
  const df64 p = two_prod(t.hi, den.hi), c = two_prod(t.hi, den.lo), e = two_prod(t.lo, den.hi);
  const df64 b = two_sum(__fsub_rn(num.hi, p.hi), -p.lo), s1 = two_sum(b.hi, num.lo), s2 = two_sum(s1.hi, -c.hi),
             s3 = two_sum(s2.hi, -e.hi);
  const float up = __fadd_rn(__fadd_rn(s1.lo, s2.lo), __fadd_rn(s3.lo, b.lo));
  const float down = __fmaf_rn(t.lo, den.lo, __fadd_rn(c.lo, e.lo));
  const float rem = __fadd_rn(s3.hi, __fsub_rn(up, down));
  return fast_two_sum(t.hi, __fmaf_rn(rem, rcp.hi, t.lo));
}
// a b with the cross terms' errors carried along.
__device__ __forceinline__ df64 df_product(df64 a, df64 b) {
  const df64 p = two_prod(a.hi, b.hi), c = two_prod(a.hi, b.lo), e = two_prod(a.lo, b.hi);
  const df64 s = two_sum(c.hi, e.hi), t = two_sum(s.hi, __fmaf_rn(a.lo, b.lo, p.lo));
  const float lo = __fadd_rn(__fadd_rn(__fadd_rn(c.lo, e.lo), s.lo), t.lo);
  return fast_two_sum(p.hi, __fadd_rn(t.hi, lo));
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
__device__ __forceinline__ df64 by_rcp(df64 num, df64 den, df64 rcp) {
  const float m = fabsf(den.hi);
  if (m > 1e-30f && m < 1e30f) return df_quotient(num, den, rcp);
  return num / den;
}
__device__ __forceinline__ double by_rcp(double num, double den, double) { return num / den; }
__device__ __forceinline__ df64 rcp_of(df64 v) { return df64(1.f) / v; }
__device__ __forceinline__ double rcp_of(double) { return 0.0; }

// Step lengths of the single-reduction iteration from (r, u), (w, u), the
// previous (r, u) and alpha and their reciprocals, which are known before the
// sums are: b = g / g_prev, a = g / (d - b g / a_prev), with one division after
// them instead of three.  Mixed path: g / a_prev beside b, not behind it.
__device__ __forceinline__ void cgf_steps(df64 g, df64 d, df64 g_prev, df64 a_prev, df64 g_rcp, df64 a_rcp, df64* a,
                                          df64* b) {
  const df64 bn = by_rcp(g, g_prev, g_rcp), ga = by_rcp(g, a_prev, a_rcp);
  *b = bn;
  *a = g / df_difference(d, df_product(bn, ga));
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
