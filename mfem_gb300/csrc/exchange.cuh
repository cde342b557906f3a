// Exchange of data between the co-resident blocks of one launch through L2:
// 16-byte records whose last word is the exchange's sequence number, written
// and read as single 128-bit accesses, so that a reader polls the record
// itself and needs no fence or flag beside it.  Every wait is bounded.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mfem_gpu {

constexpr unsigned long long kExchangeTimeoutNs = 2000000000ull;
constexpr unsigned int kExchangeMaxPolls = 1u << 24;

__device__ __forceinline__ uint4 ld_rec(const uint4* p) {
  unsigned long long a, b;
  asm volatile(
      "{\n\t.reg .b128 q;\n\t"
      "ld.relaxed.gpu.global.b128 q, [%2];\n\t"
      "mov.b128 {%0, %1}, q;\n\t}"
      : "=l"(a), "=l"(b)
      : "l"(p)
      : "memory");
  return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}
__device__ __forceinline__ void st_rec(uint4* p, uint4 v) {
  const unsigned long long a = (unsigned long long)v.x | ((unsigned long long)v.y << 32);
  const unsigned long long b = (unsigned long long)v.z | ((unsigned long long)v.w << 32);
  asm volatile(
      "{\n\t.reg .b128 q;\n\t"
      "mov.b128 q, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
      "l"(a), "l"(b)
      : "memory");
}
__device__ __forceinline__ uint4 rec_of(double v, unsigned tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return make_uint4((unsigned)b, (unsigned)(b >> 32), 0u, tag);
}
__device__ __forceinline__ double rec_double(uint4 v) {
  return __longlong_as_double((long long)((unsigned long long)v.x | ((unsigned long long)v.y << 32)));
}

__device__ __forceinline__ unsigned long long exchange_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Whether a wait of the calling warp has run out, or another block has raised
// the error flag; every 64th poll (n counts them, t0 is set on the first
// call).  Warp-uniform.
static __device__ __noinline__ bool wait_over(unsigned n, unsigned long long* t0, int* error) {
  const unsigned long long now = exchange_ns();
  if (*t0 == 0) *t0 = now;
  bool over = *(volatile int*)error != 0;
  if (now - *t0 > kExchangeTimeoutNs || n > kExchangeMaxPolls) {
    atomicExch(error, 1);
    over = true;
  }
  return __any_sync(0xffffffffu, over);
}

// Loads N records a lane and polls until all of them carry the tag, the whole
// warp in step (a lane that stopped polling early would leave the warp
// diverged for the shuffles that follow).  want: the records the lane needs;
// the others' values are not looked at.  False: the wait ran out.
template <int N, typename Ptr>
__device__ __forceinline__ bool poll_recs(uint4 (&v)[N], const Ptr& at, const bool (&want)[N], unsigned tag,
                                          int* error) {
  unsigned long long t0 = 0;
#pragma unroll 1
  for (unsigned n = 1;; ++n) {
    bool good = true;
#pragma unroll
    for (int q = 0; q < N; ++q) good = good && (!want[q] || v[q].w == tag);
    if (__all_sync(0xffffffffu, good)) return true;
    if ((n & 63u) == 0 && wait_over(n, &t0, error)) return false;
#pragma unroll
    for (int q = 0; q < N; ++q)
      if (want[q]) v[q] = ld_rec(at(q));
  }
}

// Copies of each partial sum's record: blocks poll the copy of their number
// modulo the copies, since records that every block polls queue up in L2.
// An exchange of two sums between 34 / 66 / 117 / 152 blocks alone took 2421 /
// 4956 / 7657 / 8758 cycles with one copy, 2701 / 3201 / 3392 / 3395 with
// eight (and 2422 / 2868 / 3839 / 4789 with a copy for every block); a solve's
// iteration 6.13 / 7.53 us with one / eight copies at 34 / 117 blocks against
// 6.67 with two at 34 and 8.9 with one at 117.
constexpr int kMaxCopies = 8;
__host__ __device__ constexpr int exchange_copies(int blocks) { return blocks > 40 ? kMaxCopies : 1; }

// n records of one quantity summed by the calling warp (valid in lane 0):
// lane l over records l, l + 32, ..; then a tree; 160 records in flight, so
// that a block an SM takes one wait.  Absent records are not added: a zero
// takes an addition's 66 cycles too.  ok is cleared when a wait ran out.
__device__ __forceinline__ double fetch_sum(const uint4* rec, int n, unsigned seq, int* err, bool& ok) {
  const int lane = threadIdx.x & 31;
  double v = 0.0;
  for (int i0 = 0; i0 < n && ok; i0 += 160) {
    uint4 g[5];
    bool want[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      want[j] = i0 + 32 * j + lane < n;
      if (want[j]) g[j] = ld_rec(rec + i0 + 32 * j + lane);
    }
    ok = poll_recs<5>(g, [&](int j) { return rec + i0 + 32 * j + lane; }, want, seq, err);
#pragma unroll
    for (int j = 0; j < 5; ++j)
      if (i0 + 32 * j < n) {  // warp-uniform
        const double e = want[j] ? rec_double(g[j]) : 0.0;
        v = i0 + j == 0 ? e : v + e;
      }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
    if (off < n) v += __shfl_down_sync(0xffffffffu, v, off);
  return v;
}

// num / den for a den whose correctly rounded reciprocal is at hand: one
// product and one correction of the remainder give the correctly rounded
// quotient (Markstein 1990), in 3 instead of the division's 9 latencies.  (The
// division proper, where a reciprocal or product is out of range, is a call:
// inlined, both would be computed each time.)
__device__ __noinline__ inline double quotient(double num, double den) { return num / den; }
__device__ __forceinline__ double quotient_by(double num, double den, double rcp) {
  const double q = num * rcp;
  const double v = fma(fma(-den, q, num), rcp, q);
  return isfinite(v) ? v : quotient(num, den);
}

}  // namespace mfem_gpu
