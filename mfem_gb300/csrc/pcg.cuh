// Pieces the PCG kernels share (k_rows.cu: one launch per iteration or per
// half iteration; k_resident.cu: a whole solve in one launch): vector and
// matrix access, the preconditioner, and the scalar steps of both iterations.
// Every form of an iteration calls the same functions in the same order, with
// explicit FMAs, so that its results do not depend on the form that runs it.
#pragma once
#include <cfloat>

#include "device_math.cuh"
#include "kernels.cuh"
#include "pcg_scalars.cuh"
#include "reduce.cuh"

namespace mfem_gpu {

// Three components of a row of a 4-padded vector: one 16-byte access in
// FP32, two in FP64.  kCo: the load bypasses L1 (data written by other
// blocks earlier in the same launch).
template <bool kCo>
__device__ __forceinline__ void ld3(const float* p, float v[3]) {
  const float4 t = kCo ? __ldcg(reinterpret_cast<const float4*>(p)) : *reinterpret_cast<const float4*>(p);
  v[0] = t.x;
  v[1] = t.y;
  v[2] = t.z;
}
template <bool kCo>
__device__ __forceinline__ void ld3(const double* p, double v[3]) {
  const double2 a = kCo ? __ldcg(reinterpret_cast<const double2*>(p)) : *reinterpret_cast<const double2*>(p);
  const double2 b = kCo ? __ldcg(reinterpret_cast<const double2*>(p) + 1) : reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
}
__device__ __forceinline__ void st3(float* p, const float v[3]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], 0.f);
}
__device__ __forceinline__ void st3(double* p, const double v[3]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], 0.0);
}

// Loads of data that other blocks wrote earlier in the same launch: in the
// persistent PCG (kCo) they bypass L1, which is not coherent across SMs;
// between separate launches a plain load is fine.
template <bool kCo, typename T> __device__ __forceinline__ T ldv(const T* p) {
  if constexpr (kCo) return __ldcg(p);
  else return *p;
}

// Pair w of a packed ELL slot; the column of pair 0 is stored as the
// integer's bits in the first word.
template <bool kCo>
__device__ __forceinline__ float2 ld_pair(const float* ell, size_t pair) {
  const float2* p = reinterpret_cast<const float2*>(ell) + pair;
  return kCo ? __ldcg(p) : *p;
}
template <bool kCo>
__device__ __forceinline__ double2 ld_pair(const double* ell, size_t pair) {
  const double2* p = reinterpret_cast<const double2*>(ell) + pair;
  return kCo ? __ldcg(p) : *p;
}
// L2 policies for the PCG's SpMV: the matrix is streamed once per iteration
// (evict first, no L1 allocation, read-only path), while the vectors the
// SpMV gathers at neighbouring rows are kept (evict last).  Without them the
// 115 MB matrix stream of a 1M-tet scene pushes the 4 MB vectors out of L2.
__device__ __forceinline__ unsigned long long l2_evict_first() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long l2_evict_last() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// L2 policy of the matrix stream: all lines evict-first (keep = 0), or half
// (keep = 1) or three eighths (keep = 2) of them evict-last, so that about
// that much of the matrix can stay in L2 from one iteration to the next.
template <int kKeep>
__device__ __forceinline__ unsigned long long l2_matrix_policy() {
  unsigned long long p;
  if constexpr (kKeep == 0)
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  else if constexpr (kKeep == 1)
    asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_first.b64 %0, 0.5;" : "=l"(p));
  else
    asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_first.b64 %0, 0.375;" : "=l"(p));
  return p;
}

__device__ __forceinline__ float2 ld_stream(const float* ell, size_t pair, unsigned long long pol) {
  float2 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;"
               : "=f"(v.x), "=f"(v.y) : "l"(reinterpret_cast<const float2*>(ell) + pair), "l"(pol));
  return v;
}
__device__ __forceinline__ double2 ld_stream(const double* ell, size_t pair, unsigned long long pol) {
  double2 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
               : "=d"(v.x), "=d"(v.y) : "l"(reinterpret_cast<const double2*>(ell) + pair), "l"(pol));
  return v;
}
// Gather of a row's three components with the keep policy (between
// launches only: the persistent form bypasses L1 instead).
__device__ __forceinline__ void ld3_keep(const float* p, float v[3], unsigned long long pol) {
  float4 t;
  asm volatile("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w) : "l"(p), "l"(pol));
  v[0] = t.x;
  v[1] = t.y;
  v[2] = t.z;
}
__device__ __forceinline__ void ld3_keep(const double* p, double v[3], unsigned long long pol) {
  double2 a, b;
  asm volatile("ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(a.x), "=d"(a.y) : "l"(p), "l"(pol));
  asm volatile("ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(b.x), "=d"(b.y) : "l"(p + 2), "l"(pol));
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
}
template <bool kCo, typename Real>
__device__ __forceinline__ void ld3_gather(const Real* p, Real v[3], unsigned long long pol) {
  if constexpr (kCo) ld3<true>(p, v);
  else ld3_keep(p, v, pol);
}

__device__ __forceinline__ int pair_col(float2 w) { return __float_as_int(w.x); }
__device__ __forceinline__ int pair_col(double2 w) { return (int)__double_as_longlong(w.x); }

// x of the mixed-path PCG in df64: a row is 4 float pairs (32 bytes).
struct X3 {
  df64 v[3];
};
__device__ __forceinline__ X3 zero_x3() { return X3{{df64(0.f), df64(0.f), df64(0.f)}}; }
template <bool kCo>
__device__ __forceinline__ X3 xe_load(const void* base, int row) {
  const float4* p = static_cast<const float4*>(base) + 2 * (size_t)row;
  const float4 a = kCo ? __ldcg(p) : p[0];
  const float4 b = kCo ? __ldcg(p + 1) : p[1];
  return X3{{df64(a.x, a.y), df64(a.z, a.w), df64(b.x, b.y)}};
}
__device__ __forceinline__ void xe_store(void* base, int row, const X3& x) {
  float4* p = static_cast<float4*>(base) + 2 * (size_t)row;
  p[0] = make_float4(x.v[0].hi, x.v[0].lo, x.v[1].hi, x.v[1].lo);
  p[1] = make_float4(x.v[2].hi, x.v[2].lo, 0.f, 0.f);
}

// Products of two Reals carried exactly in Ext (TwoProduct in the mixed path).
__device__ __forceinline__ df64 exact_prod(float a, float b) { return two_prod(a, b); }
__device__ __forceinline__ double exact_prod(double a, double b) { return a * b; }
// acc + a b with the exact product (one rounding in FP64).
__device__ __forceinline__ df64 acc_prod(df64 acc, float a, float b) { return acc + two_prod(a, b); }
__device__ __forceinline__ double acc_prod(double acc, double a, double b) { return fma(a, b, acc); }

// z = D^{-1} r for one row (Jacobi or 3x3 block Jacobi).
template <typename Real>
__device__ __forceinline__ void apply_prec(const SceneDev& sd, int row, const Real r[3], Real z[3]) {
  const Real* dinv = static_cast<const Real*>(sd.dinv);
  if (sd.block_jacobi) {
    const Real* D = dinv + 9 * (size_t)row;
#pragma unroll
    for (int c = 0; c < 3; ++c) z[c] = fma(D[3 * c + 2], r[2], fma(D[3 * c + 1], r[1], D[3 * c] * r[0]));
  } else {
    Real d[3];
    ld3<false>(dinv + 4 * (size_t)row, d);
#pragma unroll
    for (int c = 0; c < 3; ++c) z[c] = d[c] * r[c];
  }
}

// acc += B u for one packed ELL slot (pairs (col, a00) (a01, a02) (a10, a11)
// (a12, a20) (a21, a22)), as explicit FMA chains: every form of the fused
// iteration (registers or staged through shared memory) rounds alike.
template <typename P, typename Real>
__device__ __forceinline__ void ell_block_fma(const P& w0, const P& w1, const P& w2, const P& w3, const P& w4,
                                              const Real u[3], Real& a0, Real& a1, Real& a2) {
  a0 = fma(w1.y, u[2], fma(w1.x, u[1], fma(w0.y, u[0], a0)));
  a1 = fma(w3.x, u[2], fma(w2.y, u[1], fma(w2.x, u[0], a1)));
  a2 = fma(w4.y, u[2], fma(w4.x, u[1], fma(w3.y, u[0], a2)));
}

// A row of the two-reduction iteration's product: FP32 one chain over the
// slots; FP64 four, over the slots k = j mod 4, added up in pairs, so that the
// resident solve can give the parts of a long chain of 66-cycle instructions
// to different warps.
template <typename Real> struct RowSum;
template <> struct RowSum<float> {
  float a[3] = {0.f, 0.f, 0.f};
  template <typename P>
  __device__ __forceinline__ void add(int, const P& w0, const P& w1, const P& w2, const P& w3, const P& w4,
                                      const float u[3]) {
    ell_block_fma(w0, w1, w2, w3, w4, u, a[0], a[1], a[2]);
  }
  __device__ __forceinline__ void total(float y[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) y[c] = a[c];
  }
};
template <> struct RowSum<double> {
  double a[4][3] = {};
  template <typename P>
  __device__ __forceinline__ void add(int k, const P& w0, const P& w1, const P& w2, const P& w3, const P& w4,
                                      const double u[3]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if ((k & 3) == j) ell_block_fma(w0, w1, w2, w3, w4, u, a[j][0], a[j][1], a[j][2]);
  }
  __device__ __forceinline__ void total(double y[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) y[c] = (a[0][c] + a[1][c]) + (a[2][c] + a[3][c]);
  }
};

// u_{i+1} of a row from r_i, w_i, s_{i-1}: the same operations, in the same
// order, wherever a row's value is formed.
template <typename Real>
__device__ __forceinline__ void cgf_next(const SceneDev& sd, int row, const Real r[3], const Real w[3],
                                         const Real sp[3], Real a, Real b, Real s[3], Real rn[3],
                                         Real u[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    s[c] = fma(b, sp[c], w[c]);
    rn[c] = fma(-a, s[c], r[c]);
  }
  apply_prec<Real>(sd, row, rn, u);
}

// ------------------------------------------------ scalars of a solve ---
// The inner products and step lengths live in the path's high precision
// (float-float or double) in 8-byte slots of SceneScalars.
template <typename E> __device__ __forceinline__ E sc_get(const double* p) { return Slot<E>::get(p); }
template <typename E> __device__ __forceinline__ void sc_put(double* p, E v) { Slot<E>::put(p, v); }
__device__ __forceinline__ bool is_nan(df64 v) { return v.hi != v.hi; }
__device__ __forceinline__ bool is_nan(double v) { return v != v; }
__device__ __forceinline__ bool is_zero(df64 v) { return v.hi == 0.f; }
__device__ __forceinline__ bool is_zero(double v) { return v == 0.0; }
__device__ __forceinline__ double to_step(double v) { return v; }

// The stopping test |r|^2 < max(tol^2 |b|^2, DBL_MIN).  The mixed path forms
// the threshold in FP64 once a solve, for any tolerance, and keeps it as two
// floats: the nearest float and the rest rounded up.  A float-float |r|^2 then
// lies below it exactly when the pairs compare so, with no FP64 instruction an
// iteration: where the first floats differ they decide, and a float lies below
// the rest when it lies below the next float above.  (A threshold past FP32's
// range becomes (inf, -inf), which every finite sum meets, one below it (0,
// 1.4e-45), which only zero meets.)
__device__ __forceinline__ double cg_threshold_fp64(const SceneDev& sd, double rr0) {
  return ::fmax(sd.cg_tol * sd.cg_tol * rr0, DBL_MIN);
}
__device__ __forceinline__ float2 cg_threshold(const SceneDev& sd, df64 rr0) {
  const double t = cg_threshold_fp64(sd, rr0.to_double());
  const float hi = float(t);
  return make_float2(hi, __double2float_ru(t - double(hi)));
}
__device__ __forceinline__ float2 cg_threshold(const SceneDev&, double) { return make_float2(0.f, 0.f); }
__device__ __forceinline__ bool cg_meets(const SceneDev&, float2 thr, df64 rr, df64) {
  return rr < df64(thr.x, thr.y);
}
__device__ __forceinline__ bool cg_meets(const SceneDev& sd, float2, double rr, double rr0) {
  return rr < cg_threshold_fp64(sd, rr0);
}
__device__ __forceinline__ double cg_rel(df64 rr, df64 rr0) { return double(sqrtf(rr.hi / rr0.hi)); }
__device__ __forceinline__ double cg_rel(double rr, double rr0) { return ::sqrt(rr / rr0); }

// ---------------------------------------- verified stop (mixed path) ---
// In FP32 the single-reduction recurrences drift: the recursive residual
// meets the tolerance while the true |b - A x| / |b| sits several times
// above it (x itself rounded to FP32 floors it near eps32 |A||x| / |b|).
// So when the recursion says "converged", the mixed path verifies before it
// stops, in three further launches of the same kernel (the scene's
// cgf_phase selects the work; the iteration count does not move):
//   1  r = b - A (x_e + x), with each FP32 matrix entry times the df64
//      x_e + x as an exact product summed in df64 (the reliable residual);
//      u = M^-1 r;
//   2  x_e += x, x = 0 (the FP32 x restarts as a correction, so its
//      rounding shrinks with what is left to solve); w = A u and s = A p
//      (the recursions' drift starts again from zero); the inner products
//      of the true residual.  If it meets the tolerance: phase 3.
//      Otherwise the recursion continues from the replaced r, w and s:
//      the next direction u + b p is made A-conjugate to p directly (b =
//      -(A p, u) / (p, A p)), because the drifted recursion's
//      gamma_prev no longer describes the true residual, and a from the
//      exact (p_new, A p_new).  After kCgfRounds failed verifications the
//      next recursive stop is accepted as it is;
//   3  x_e += x, and x = round(x_e) for the readers of the solution; stop.
// A stop on max_iterative_solver_iters or a non-finite residual also goes
// through phase 3, so the solution is always x_e + x.

// The finalizer's part for the mixed path (thread 0 of the scene's last tile).
constexpr int kCgfRounds = 4;
__device__ __forceinline__ void cgf_verify_step(const SceneDev& sd, BatchCounters* ctrs, df64 rr, df64 g,
                                                df64 d, df64 su, df64 ps, int it) {
  SceneScalars* sc = sd.sc;
  const int ph = sc->cgf_phase;
  if (ph == 1) {
    sc->cgf_phase = 2;
    return;
  }
  if (ph == 3 || *(volatile int*)&ctrs->error) {
    sc->cg_total += sc->cg_iter;
    sc->cg_active = 0;
    sc->nph = kPhLocal;
    atomicSub(&ctrs->cg_active, 1);
    return;
  }
  const df64 rr0 = sc_get<df64>(&sc->cg_rhs_norm2);
  sc->cg_err = cg_rel(rr, rr0);
  if (is_nan(rr)) {
    sc->status = 4;
    sc->cgf_phase = 3;
    return;
  }
  if (cg_meets(sd, sc->cg_thr, rr, rr0)) {
    // phase 0: the recursion's residual passes, verify it (unless the
    // verifications are used up); phase 2: the true residual passes, write
    // the solution
    sc->cgf_phase = (ph == 0 && sc->cgf_rounds < kCgfRounds) ? 1 : 3;
    return;
  }
  df64 bn, an;
  if (ph == 2) {
    // A failed verification.  The recursion's gamma had drifted below the
    // true residual's, so b = gamma / gamma_prev would be far too large; su
    // and ps come from phase 2's exact A p.
    sc->cgf_rounds += 1;
    cgf_restart_steps(g, d, su, ps, &an, &bn);
  } else {
    const df64 g_prev = sc_get<df64>(&sc->cgf_gamma[0]), a_prev = sc_get<df64>(&sc->alpha);
    cgf_steps(g, d, g_prev, a_prev, rcp_of(g_prev), rcp_of(a_prev), &an, &bn);
  }
  sc_put(&sc->beta, bn);
  sc->beta_f = to_step(bn);
  sc_put(&sc->alpha, an);
  sc->alpha_f = to_step(an);
  sc_put(&sc->cgf_gamma[0], g);
  sc->cg_iter = it + 1;
  sc->cgf_phase = 0;
  if (it + 1 >= sd.max_cg) {
    sc->cg_status = 5;  // MFEM_ERR_CG_MAXITER
    sc->cgf_phase = 3;
  }
}

}  // namespace mfem_gpu
