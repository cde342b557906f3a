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

}  // namespace mfem_gpu
