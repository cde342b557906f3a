// PCG solves in one launch with the matrix resident in shared memory.
//
// A system of up to some ten thousand block rows has a matrix of at most
// 34 MB: it fits the SMs' shared memory together, or at worst the L2, and an
// iteration moves almost nothing.  What one launch per half iteration
// (k_cg_spmv, k_cg_update) or per iteration (k_cgf_iter) then costs is the
// chain of latencies: launch boundaries, a row's slots walked one after
// another (column -> gather -> FMA), tile tickets, a serial finalizer.  Here
// each block owns up to sixteen 32-row slices for the whole solve and
//   * copies its slices' blocks to shared memory once, as nine planes of 32
//     lanes per slot, and keeps its rows' vectors in registers;
//   * knows its halo, the distinct columns outside its rows (built by the
//     host), and once per iteration fetches one vector at them, all columns
//     in flight together, updates its copy of the multiplied vector with the
//     owner's own operations, and multiplies out of shared memory;
//   * exchanges data through L2 without fences, flags or atomics: a row's
//     vector and a block's partial sums are 16-byte records whose last word
//     is the exchange's sequence number, written and read as single 128-bit
//     accesses, so a reader polls the record itself.  Every block sums all
//     partials in the same fixed order and takes the same decisions.
// The arithmetic, the order of every sum included, is that of the launches
// it replaces (pcg.cuh), so the results are bitwise the same.
// k_cgr_split (mixed path) and k_cgr_split64 run the two-reduction iteration,
// k_cgr_fused the single-reduction one, and k_cgr_wide that one for systems
// that outgrow shared memory, whose matrix it streams.
//
// A record is overwritten only after everybody has read it: partials and the
// single-reduction form's vector alternate between two buffers by the
// exchange's parity, and a block writes exchange k + 2 only after it has read
// k + 1 from every block, which each wrote after reading k; the two-reduction
// form's vector has a second exchange between its reading and its writing.
// Sequence numbers go on from launch to launch (CgrArgs::seq).
//
// Every wait is bounded: after kExchangeTimeoutNs the block raises ctrs->error and
// leaves, as do the others when they see the flag or time out themselves; the
// host reports MFEM_ERR_TIMEOUT.  The launch is cooperative: all blocks are
// co-resident, the exchange needs them all.
#include <new>
#include <type_traits>

#include "async_copy.cuh"
#include "exchange.cuh"
#include "pcg.cuh"
#include "resident.cuh"

namespace mfem_gpu {

namespace {

using mfem_gpu::rec_of;
__device__ __forceinline__ uint4 rec_of(df64 v, unsigned tag) {
  return make_uint4(__float_as_uint(v.hi), __float_as_uint(v.lo), 0u, tag);
}
template <typename E> __device__ __forceinline__ E rec_val(uint4 v);
template <> __device__ __forceinline__ df64 rec_val<df64>(uint4 v) {
  return df64(__uint_as_float(v.x), __uint_as_float(v.y));
}

__device__ __forceinline__ df64 shfl_to(df64 v, int lane) {
  return df64(__shfl_sync(0xffffffffu, v.hi, lane), __shfl_sync(0xffffffffu, v.lo, lane));
}

template <typename E, int NQ, int kFrom>
__device__ __forceinline__ void tree(E (&v)[NQ]) {
#pragma unroll
  for (int off = kFrom; off > 0; off >>= 1)
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = radd(v[q], shfl_down(v[q], off));
}

struct CgrShared {
  double part[2][3][kCgrMaxSlices];  // the block's slice sums
  double red[2][3][8];               // warp sums of the tiles
  int late;                          // a wait of scene_total ran out (cleared by the kernel)
};

// Sums over the scene's rows, the same in every thread of every block.  v
// holds each lane's values in the lead warps (one per slice, `sl` its number
// in the block); the order is that of tile_partials and scene_sums: a tree
// over a slice's 32 rows, a tree over the 8 slices of a tile, each thread over
// tiles i, i + 256, .., a tree over 32 such sums, a tree over 8.  (Their
// trees over absent entries only add zeros.)  A block sends the sums of its
// one or two tiles, a scene of one block nothing.  `ahead` runs once the
// other blocks' sums have come in, before the last of the adding: loads issued
// there are under way meanwhile; `during` before, while the sums travel.
// kLead: only the first warp wants the sums (the others have them of more than
// 32 records).  False: a wait ran out; of up to 32 records for the warps whose wait it was,
// of more for the whole block.
template <typename E, int NQ, bool kLead = false, typename F, typename G>
__device__ __forceinline__ bool scene_total(const CgrArgs& A, const CgrBlock& B, CgrShared& S, bool lead, int sl,
                                            unsigned seq, E (&v)[NQ], const F& ahead, const G& during) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int par = seq & 1;
  const int copies = exchange_copies(B.nblk);
  const size_t cstride = 3 * (size_t)A.nrec_total;
  uint4* rec = A.recs + par * kMaxCopies * cstride + B.rec0;
  // lane 0's value as every copy of record i of quantity q (the whole warp)
  auto send = [&](int q, int i, E val) {
    const E a = shfl_to(val, 0);
    if (lane < copies) st_rec(rec + lane * cstride + (size_t)q * A.nrec_total + i, rec_of(a, seq));
  };
  if (lead) tree<E, NQ, 16>(v);
  if (lead && lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) Slot<E>::put(&S.part[par][q][sl], v[q]);
  __syncthreads();
  const int nt = (B.nsl + kCgrTile - 1) / kCgrTile;  // 1 or 2
  if (B.nblk == 1 && kLead && warp > 0) return true;
  if (B.nblk == 1) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = lane < B.nsl ? Slot<E>::sget(&S.part[par][q][lane]) : E(0);
    tree<E, NQ, 4>(v);  // the tiles' sums in lanes 0 and 8
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (nt > 1) v[q] = radd(v[q], shfl_to(v[q], 8));
      v[q] = shfl_to(v[q], 0);
    }
    during();
    ahead();
    return true;
  }
  if (warp < NQ * nt) {
    const int q = warp / nt, t = warp % nt, at = kCgrTile * t + lane;
    E a[1] = {lane < kCgrTile && at < B.nsl ? Slot<E>::sget(&S.part[par][q][at]) : E(0)};
    tree<E, 1, 4>(a);
    send(q, B.rec + t, a[0]);
  }
  during();
  const int n = B.nrec;
  // the sums of record i (0 for lanes without one), the warp in step
  auto fetch = [&](int i, E (&a)[NQ]) -> bool {
    uint4 w[NQ];
    bool want[NQ];
    const uint4* src = rec + (blockIdx.x % copies) * cstride + min(i, n - 1);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      want[q] = i < n;
      w[q] = ld_rec(src + (size_t)q * A.nrec_total);
    }
    const bool ok = poll_recs<NQ>(w, [&](int q) { return src + (size_t)q * A.nrec_total; }, want, seq, &A.ctrs->error);
#pragma unroll
    for (int q = 0; q < NQ; ++q) a[q] = i < n ? rec_val<E>(w[q]) : E(0);
    return ok;
  };
  if (n <= 32) {
    // every warp for itself, no block barrier
    if (kLead && warp > 0) {
      ahead();
      return true;
    }
    E a[NQ];
    if (!fetch(lane, a)) return false;
    ahead();
    tree<E, NQ, 16>(a);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = shfl_to(a[q], 0);
    return true;
  }
  E s[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) s[q] = E(0);
  bool ok = true;
  if (warp < 8) {
    for (int i0 = 32 * warp; i0 < n && ok; i0 += 256) {
      E a[NQ];
      ok = fetch(i0 + lane, a);
#pragma unroll
      for (int q = 0; q < NQ; ++q) s[q] = radd(s[q], a[q]);
    }
    // (the warps wait for different records: a wait that ran out shows in the
    // sums, so that all warps leave or none; __syncthreads_and took 1% of a step)
    if (!ok) {
      S.late = 1;
#pragma unroll
      for (int q = 0; q < NQ; ++q) s[q] = E(__int_as_float(0x7fffffff));
    }
    tree<E, NQ, 16>(s);
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < NQ; ++q) Slot<E>::put(&S.red[par][q][warp], s[q]);
  }
  __syncthreads();
  ahead();
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = lane < 8 ? Slot<E>::sget(&S.red[par][q][lane]) : E(0);
  tree<E, NQ, 4>(v);
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = shfl_to(v[q], 0);
  return !(is_nan(v[0]) && S.late);
}

// The block's slices in shared memory: nine planes (row-major 3x3 entries) of
// 32 lanes per resident slot, and each slot's local column indices.
template <typename Real> struct CgrMatrix {
  const Real* mat;       // this warp's slice: + 288 k + 32 e + lane
  const uint16_t* li;    // + 32 k + lane
  int res, len;          // resident and all slots of the slice
  const Real* gell;      // the slice in the packed global layout (pairs from 5 soff)
  const uint16_t* gli;
  int soff;
};

template <typename Real>
__device__ __forceinline__ CgrMatrix<Real> cgr_load_matrix(const CgrArgs& A, const CgrBlock& B, const SceneDev& sd,
                                                           int sl, unsigned char* smem, unsigned char** rest) {
  using P = typename std::conditional<sizeof(Real) == 4, float2, double2>::type;
  const int soff0 = sd.slice_off[B.slice0];
  int slots = 0;
  for (int s = 0; s < B.nsl; ++s)
    slots += min(B.kres, (sd.slice_off[B.slice0 + s + 1] - sd.slice_off[B.slice0 + s]) >> 5);
  Real* mat = reinterpret_cast<Real*>(smem);
  uint16_t* li = reinterpret_cast<uint16_t*>(mat + (size_t)slots * 288);
  *rest = reinterpret_cast<unsigned char*>(li + (size_t)slots * 32);
  CgrMatrix<Real> M{};
  int at = 0;
  for (int s = 0; s < B.nsl; ++s) {
    const int soff = sd.slice_off[B.slice0 + s], len = (sd.slice_off[B.slice0 + s + 1] - soff) >> 5;
    const int res = min(B.kres, len);
    const P* src = static_cast<const P*>(sd.ell) + 5 * (size_t)soff;
    Real* dst = mat + (size_t)at * 288;
#pragma unroll 4
    for (int i = threadIdx.x; i < res * 160; i += blockDim.x) {
      const P v = src[i];
      const int k = i / 160, w = (i - 160 * k) >> 5, l = i & 31;
      Real* d = dst + 288 * k + l;
      if (w == 0) {
        d[0] = v.y;
      } else {
        d[32 * (2 * w - 1)] = v.x;
        d[32 * (2 * w)] = v.y;
      }
    }
    const uint16_t* gl = A.lidx + B.loff + (soff - soff0);
    for (int i = threadIdx.x; i < res * 32; i += blockDim.x) li[32 * at + i] = gl[i];
    if (s == sl) {
      M.mat = dst;
      M.li = li + 32 * at;
      M.res = res;
      M.len = len;
      M.gell = static_cast<const Real*>(sd.ell);
      M.gli = gl;
      M.soff = soff;
    }
    at += res;
  }
  return M;
}

// acc += (row of A) u, slots in order; u: float4 per local index.
__device__ __forceinline__ void cgr_multiply(const CgrMatrix<float>& M, const float4* u, float (&acc)[3]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int k = 0; k < M.res; ++k) {
    const float4 p = u[M.li[32 * k + lane]];
    const float* m = M.mat + 288 * k + lane;
    acc[0] = fma(m[64], p.z, fma(m[32], p.y, fma(m[0], p.x, acc[0])));
    acc[1] = fma(m[160], p.z, fma(m[128], p.y, fma(m[96], p.x, acc[1])));
    acc[2] = fma(m[256], p.z, fma(m[224], p.y, fma(m[192], p.x, acc[2])));
  }
#pragma unroll 2
  for (int k = M.res; k < M.len; ++k) {
    const size_t q = ell_pair(M.soff, k, lane, 0);
    const float2 w0 = ld_pair<false>(M.gell, q), w1 = ld_pair<false>(M.gell, q + 32),
                 w2 = ld_pair<false>(M.gell, q + 64), w3 = ld_pair<false>(M.gell, q + 96),
                 w4 = ld_pair<false>(M.gell, q + 128);
    const float4 p4 = u[M.gli[32 * k + lane]];
    const float p[3] = {p4.x, p4.y, p4.z};
    ell_block_fma(w0, w1, w2, w3, w4, p, acc[0], acc[1], acc[2]);
  }
}
// A solve that ended on a wait that ran out: later launches use other tags.
__device__ __forceinline__ void cgr_abort(const CgrArgs& A, const CgrBlock& B) {
  if ((threadIdx.x & 31) == 0) atomicAdd(A.seq + B.scene, 0x100000u);
}

constexpr int kHaloRegs = 4;  // halo columns a thread keeps in registers

// ------------------------------------------------ two-reduction form ---
// Eigen's iteration, as k_cg_spmv, k_cg_update and k_cg_replace run it:
//   p = z + beta p;  Ap;  (p, Ap) -> alpha;  x += alpha p;  r -= alpha Ap;
//   z = D^-1 r;  (r, r), (r, z) -> the stopping test and beta;
// the exchanged vector is z, and each block keeps p at its halo.  Mixed path.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1) k_cgr_split(const CgrArgs A) {
  using E = df64;
  extern __shared__ __align__(16) unsigned char cgr_smem_raw[];
  __shared__ CgrShared S;
  const CgrBlock B = A.blocks[blockIdx.x];
  const SceneDev& sd = A.sds[B.scene];
  SceneScalars* sc = sd.sc;
  if (!sc->cg_active) return;
  unsigned seq = __ldcg(A.seq + B.scene);
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  if (threadIdx.x == 0) S.late = 0;
  const bool roww = sl < B.nsl;
  const int row = 32 * (B.slice0 + sl) + lane;
  const bool live = roww && row < sd.nf;
  const int own = 32 * B.nsl, mine = 32 * sl + lane;
  unsigned char* rest;
  const CgrMatrix<float> M = cgr_load_matrix<float>(A, B, sd, sl, cgr_smem_raw, &rest);
  float4* vec = reinterpret_cast<float4*>(rest);  // p at the own rows and the halo
  // the first halo columns of each thread, and their records under way
  int hc[kHaloRegs];
  bool hw[kHaloRegs];
  uint4 hv[kHaloRegs];
#pragma unroll
  for (int j = 0; j < kHaloRegs; ++j) {
    const int h = threadIdx.x + j * kThreads;
    hw[j] = h < B.nh;
    hc[j] = hw[j] ? A.h_col[B.hoff + h] : 0;
    if (hw[j])
      hv[j] = *reinterpret_cast<const uint4*>(static_cast<const float*>(sd.cg_z) + 4 * (size_t)hc[j]);
  }
  auto halo_ahead = [&]() {
#pragma unroll
    for (int j = 0; j < kHaloRegs; ++j)
      if (hw[j]) hv[j] = ld_rec(A.pub + B.row0 + hc[j]);
  };
  auto nothing = []() {};

  const size_t k4 = 4 * (size_t)row;
  float r[3], z[3], p[3], acc[3], dv[9];
  X3 xe = zero_x3();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    r[c] = live ? static_cast<const float*>(sd.cg_r)[k4 + c] : 0.f;
    z[c] = live ? static_cast<const float*>(sd.cg_z)[k4 + c] : 0.f;
    p[c] = acc[c] = 0.f;
  }
#pragma unroll
  for (int c = 0; c < 9; ++c)
    dv[c] = !live ? 0.f
                  : sd.block_jacobi ? static_cast<const float*>(sd.dinv)[9 * (size_t)row + c]
                                    : (c < 3 ? static_cast<const float*>(sd.dinv)[k4 + c] : 0.f);
  const bool block_jacobi = sd.block_jacobi != 0;
  // apply_prec with the row's entries in registers
  auto precond = [&](const float (&rv)[3], float (&zv)[3]) {
    if (block_jacobi) {
#pragma unroll
      for (int c = 0; c < 3; ++c) zv[c] = fma(dv[3 * c + 2], rv[2], fma(dv[3 * c + 1], rv[1], dv[3 * c] * rv[0]));
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) zv[c] = dv[c] * rv[c];
    }
  };
  E rz = sc_get<E>(&sc->rz), rz_prev = rz;
  const E rr0 = sc_get<E>(&sc->cg_rhs_norm2);
  const float2 thr = sc->cg_thr;
  E rr = rr0;
  float beta = 0.f;
  E alphaE = E(0), betaE = E(0), rz_rcp = E(0);
  int it = 0, status = 0, cg_status = 0;
  unsigned ztag = 0;

  auto publish_z = [&](unsigned tag) {
    if (live && B.nblk > 1)
      st_rec(A.pub + B.row0 + row,
             make_uint4(__float_as_uint(z[0]), __float_as_uint(z[1]), __float_as_uint(z[2]), tag));
  };

  for (;;) {
    const bool first = it == 0;
    // ---- p = z + beta p: own rows, then the halo
    if (roww) {
#pragma unroll
      for (int c = 0; c < 3; ++c) p[c] = first ? z[c] : fma(beta, p[c], z[c]);
      vec[mine] = make_float4(p[0], p[1], p[2], 0.f);
    }
    bool ok = true;
    float4* ph = vec + own;
    auto put = [&](int h, const uint4& v) {
      const float z0 = __uint_as_float(v.x), z1 = __uint_as_float(v.y), z2 = __uint_as_float(v.z);
      const float4 o = ph[h];
      ph[h] = first ? make_float4(z0, z1, z2, 0.f)
                    : make_float4(fma(beta, o.x, z0), fma(beta, o.y, z1), fma(beta, o.z, z2), 0.f);
    };
    if (!first)
      ok = poll_recs<kHaloRegs>(hv, [&](int j) { return A.pub + B.row0 + hc[j]; }, hw, ztag, &A.ctrs->error) && ok;
#pragma unroll
    for (int j = 0; j < kHaloRegs; ++j)
      if (hw[j]) put(threadIdx.x + j * kThreads, hv[j]);
    for (int h0 = 32 * sl + kHaloRegs * kThreads; h0 < B.nh; h0 += kThreads) {
      const int h = h0 + lane;
      const bool want[1] = {h < B.nh};
      const int col = want[0] ? __ldg(A.h_col + B.hoff + h) : 0;
      const uint4* src = first ? reinterpret_cast<const uint4*>(static_cast<const float*>(sd.cg_z) + 4 * (size_t)col)
                               : A.pub + B.row0 + col;
      uint4 v[1] = {ld_rec(src)};
      if (!first) ok = poll_recs<1>(v, [&](int) { return src; }, want, ztag, &A.ctrs->error) && ok;
      if (want[0]) put(h, v[0]);
    }
    if (!__syncthreads_and(ok)) {
      cgr_abort(A, B);
      return;
    }
    // ---- Ap, (p, Ap)
    E d1[1] = {E(0)};
    if (roww) {
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] = 0.f;
      cgr_multiply(M, vec, acc);
    }
    if (live) {
#pragma unroll
      for (int c = 0; c < 3; ++c) d1[0] = acc_prod(d1[0], p[c], acc[c]);
    }
    if (!scene_total<E, 1>(A, B, S, roww, sl, seq, d1, nothing, [&]() { rz_rcp = E(1.f) / rz; })) {
      cgr_abort(A, B);
      return;
    }
    ++seq;
    alphaE = rz / d1[0];
    const float alpha = to_step(alphaE);
    // ---- x, r, z, (r, r), (r, z)
    const bool replace = (it + 1) % kCgReplace == 0;
    E d2[2] = {E(0), E(0)};
    if (live) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        xe.v[c] = xe.v[c] + two_prod(alpha, p[c]);
        r[c] = fma(-alpha, acc[c], r[c]);
        d2[0] = acc_prod(d2[0], r[c], r[c]);
      }
      if (replace) {
        xe_store(sd.cg_xe, row, xe);
        __threadfence();
      }
      precond(r, z);
#pragma unroll
      for (int c = 0; c < 3; ++c) d2[1] = acc_prod(d2[1], r[c], z[c]);
      if (!replace) publish_z(seq);
    }
    if (replace) __syncthreads();  // every row's x_e is visible before the block's sums
    if (!scene_total<E, 2>(A, B, S, roww, sl, seq, d2, halo_ahead, nothing)) {
      cgr_abort(A, B);
      return;
    }
    ztag = seq;
    ++seq;
    rr = d2[0];
    bool stop = false;
    if (cg_meets(sd, thr, rr, rr0)) {
      stop = true;
    } else {
      betaE = by_rcp_step(d2[1], rz, rz_rcp);
      rz_prev = rz;
      rz = d2[1];
      it = it + 1;
      if (it >= sd.max_cg) {
        stop = true;
        cg_status = 5;  // MFEM_ERR_CG_MAXITER
      }
    }
    if (is_nan(rr)) {
      stop = true;
      status = 4;
    }
    if (stop) break;
    if (replace) {
      // ---- r = b - A x with x in df64 (k_cg_replace)
      __syncwarp();
      __threadfence();
      E d3[2] = {E(0), E(0)};
      if (live) {
        df64 ax[3] = {df64(0.f), df64(0.f), df64(0.f)};
#pragma unroll 4
        for (int k = 0; k < M.len; ++k) {
          const size_t q = ell_pair(M.soff, k, lane, 0);
          const float* ell = static_cast<const float*>(sd.ell);
          const float2 w0 = ld_pair<false>(ell, q), w1 = ld_pair<false>(ell, q + 32),
                       w2 = ld_pair<false>(ell, q + 64), w3 = ld_pair<false>(ell, q + 96),
                       w4 = ld_pair<false>(ell, q + 128);
          const X3 xc = xe_load<true>(sd.cg_xe, pair_col(w0));
          const float a[9] = {w0.y, w1.x, w1.y, w2.x, w2.y, w3.x, w3.y, w4.x, w4.y};
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const float aij = a[3 * i + j];
              ax[i] = ax[i] + two_prod(aij, xc.v[j].hi) + df64(aij * xc.v[j].lo);
            }
        }
        float b[3];
        ld3<false>(static_cast<const float*>(sd.rhs) + k4, b);
#pragma unroll
        for (int c = 0; c < 3; ++c) r[c] = Ext<float>::to_real(df64(b[c]) - ax[c]);
        precond(r, z);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          d3[0] = acc_prod(d3[0], r[c], r[c]);
          d3[1] = acc_prod(d3[1], r[c], z[c]);
        }
        publish_z(seq);
      }
      if (!scene_total<E, 2>(A, B, S, roww, sl, seq, d3, halo_ahead, nothing)) {
        cgr_abort(A, B);
        return;
      }
      ztag = seq;
      ++seq;
      rr = d3[0];
      if (cg_meets(sd, thr, rr, rr0) || is_nan(rr)) {
        if (is_nan(rr)) status = 4;
        it = it - 1;  // as in Eigen, the iteration that meets the threshold is not counted
        break;
      }
      betaE = by_rcp_step(d3[1], rz_prev, rz_rcp);
      rz = d3[1];
    }
    beta = to_step(betaE);
  }
  // ---- the solution and the scene's scalars
  if (live) {
    float xf[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) xf[c] = Ext<float>::to_real(xe.v[c]);
    st3(static_cast<float*>(sd.cg_x) + k4, xf);
    xe_store(sd.cg_xe, row, xe);
  }
  if (B.rec == 0 && threadIdx.x == 0) {
    sc_put(&sc->alpha, alphaE);
    sc_put(&sc->beta, betaE);
    sc_put(&sc->rz, rz);
    sc_put(&sc->rz_prev, rz_prev);
    sc->cg_err = cg_rel(rr, rr0);
    sc->cg_iter = it;
    sc->cg_total += it;
    if (status) sc->status = status;
    if (cg_status) sc->cg_status = cg_status;
    sc->cg_active = 0;
    sc->nph = kPhLocal;
    atomicSub(&A.ctrs->cg_active, 1);
    A.seq[B.scene] = seq;
  }
}

// The FP64 form.  What bounds it is the FP64 pipe, which takes a warp's
// instruction every 17 to 19 cycles of the SM (and 66 for the next one of the
// same warp, 576 for a division): a block has one slice, or two or four where
// there are more slices than SMs, and always twelve warps, one per slice,
// component and part of the slots (4, 2 or 1 parts: the slots k = j mod 4 are
// four sums, see RowSum); the warps of part 0 own the rows' components.  A
// slice's sums, the adding of the other blocks' and the scalars are one warp's
// each, and the quotient by a number known before is a product with its
// reciprocal, corrected (quotient_by).  An iteration at 90 / 1300 rows: 7.9 /
// 8.1 us, against 10.2 / 11.5 with a slice's component in one warp and the sums
// and scalars in every warp, and 34 / 38 in k_cg_solve.  Of the 15,600 cycles
// at 1300 rows the product is 3400 (its 180 warp instructions a slice at the
// pipe's rate), the two exchanges 5000, trees and divisions 4000.
constexpr int kThreads64 = 384;
__global__ void __launch_bounds__(kThreads64, 1) k_cgr_split64(const CgrArgs A) {
  extern __shared__ __align__(16) unsigned char cgr_smem_raw[];
  __shared__ double part[2][kCgrMaxSpb64], tile[2][kCgrMaxTiles64], tot[2], step[2], rcp;
  __shared__ int flags;  // 1: a wait ran out
  const CgrBlock B = A.blocks[blockIdx.x];
  const SceneDev& sd = A.sds[B.scene];
  SceneScalars* sc = sd.sc;
  if (!sc->cg_active) return;
  unsigned seq = __ldcg(A.seq + B.scene);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int parts = B.spb >= 4 ? 1 : 4 / B.spb;
  const int comp = warp % 3, sl = warp / 3 / parts, pt = warp / 3 % parts;
  const bool roww = sl < B.nsl, owner = roww && pt == 0;
  const int row = 32 * (B.slice0 + sl) + lane;
  const bool live = owner && row < sd.nf;
  const int own = 32 * B.nsl, mine = 32 * sl + lane;
  unsigned char* rest;
  const CgrMatrix<double> M = cgr_load_matrix<double>(A, B, sd, sl, cgr_smem_raw, &rest);
  double* vec = reinterpret_cast<double*>(rest);  // p at the own rows and the halo, 3 each
  double* ex = vec + 3 * (own + B.nh);            // [2][slice][3][32]: y / r, z
  double* sums = ex + 192 * B.nsl;                // [3][slice][3][32]: the products of parts 1 ..
  int* err = &A.ctrs->error;
  const int ex_at = 96 * sl + 32 * comp + lane;

  // the halo's entries (column, component) of this thread: the first in registers
  constexpr int kHalo = 3;
  int hc[kHalo];
  bool hw[kHalo];
  uint4 hv[kHalo];
#pragma unroll
  for (int j = 0; j < kHalo; ++j) {
    const int i = threadIdx.x + j * kThreads64;
    hw[j] = i < 3 * B.nh;
    hc[j] = hw[j] ? 3 * (B.row0 + A.h_col[B.hoff + i / 3]) + i % 3 : 0;
  }
  for (int i = threadIdx.x; i < 3 * B.nh; i += kThreads64)
    vec[3 * own + i] = static_cast<const double*>(sd.cg_z)[4 * (size_t)A.h_col[B.hoff + i / 3] + i % 3];
  auto halo_ahead = [&]() {
#pragma unroll
    for (int j = 0; j < kHalo; ++j)
      if (hw[j]) hv[j] = ld_rec(A.pub + hc[j]);
  };

  const size_t k4 = 4 * (size_t)row;
  const bool block_jacobi = sd.block_jacobi != 0;
  double r = 0.0, z = 0.0, p = 0.0, x = 0.0, y = 0.0, dv[3] = {0.0, 0.0, 0.0};
  if (live) {
    r = static_cast<const double*>(sd.cg_r)[k4 + comp];
    z = static_cast<const double*>(sd.cg_z)[k4 + comp];
    const double* dinv = static_cast<const double*>(sd.dinv);
    if (block_jacobi) {
#pragma unroll
      for (int c = 0; c < 3; ++c) dv[c] = dinv[9 * (size_t)row + 3 * comp + c];
    } else {
      dv[0] = dinv[k4 + comp];
    }
  }
  double rz = sc_get<double>(&sc->rz), rz_prev = rz, beta = 0.0;
  const double rr0 = sc_get<double>(&sc->cg_rhs_norm2);
  // (every FP64 instruction of all twelve warps takes 230 cycles of the pipe,
  // comparisons too: a sum of squares or NaN compares like its bits)
  const unsigned long long thr = __double_as_longlong(::fmax(sd.cg_tol * sd.cg_tol * rr0, DBL_MIN));  // as cg_meets
  constexpr unsigned long long kInf = 0x7ff0000000000000ull;
  double rr = rr0, alpha = 0.0;
  const int max_cg = sd.max_cg;
  int it = 0, status = 0, cg_status = 0;
  unsigned ztag = 0;
  if (threadIdx.x == 0) flags = 0;

  // A slice's sum of the lanes' e (the whole warp), as tile_partials adds them.
  auto slice_sum = [&](int q, double e) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) e += shfl_down(e, off);
    if (lane == 0) part[q][sl] = e;
    return e;
  };
  // The scene's sums of nq quantities in tot[], the slices' in part[][]: slices
  // to tiles of eight, tiles i, i + 256, .. (there are fewer), a tree over 32
  // tiles, a tree over 8 such sums; absent entries are zeros.  `beside`: the
  // last warp's, during the wait; `then(q, sum)`: lane 0's of the warp that has
  // the sum.  False: a wait ran out.
  auto total = [&](int nq, auto beside, auto then) -> bool {
    const int par = seq & 1, n = B.nrec, copies = exchange_copies(B.nblk);
    const size_t cstride = 3 * (size_t)A.nrec_total;
    uint4* rec = A.recs + par * kMaxCopies * cstride + B.rec0;
    __syncthreads();
    if (B.nblk > 1 && warp < nq * B.nsl) {
      const int q = warp / B.nsl, t = warp % B.nsl;
      const double v = part[q][t];
      if (lane < copies) st_rec(rec + lane * cstride + (size_t)q * A.nrec_total + B.rec + t, rec_of(v, seq));
    }
    if (warp == kThreads64 / 32 - 1) beside();
    const uint4* src = rec + (blockIdx.x % copies) * cstride;
    const int chunks = (n + 31) / 32;
    for (int job = warp; job < nq * chunks; job += kThreads64 / 32) {
      const int q = job / chunks, i = 32 * (job % chunks) + lane;
      double v = 0.0;
      if (B.nblk > 1) {
        const uint4* at = src + (size_t)q * A.nrec_total + min(i, n - 1);
        uint4 w[1] = {ld_rec(at)};
        const bool want[1] = {i < n};
        if (!poll_recs<1>(w, [&](int) { return at; }, want, seq, err) && lane == 0) atomicOr(&flags, 1);
        v = i < n ? rec_double(w[0]) : 0.0;
      } else if (i < n) {
        v = part[q][i];
      }
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) v += shfl_down(v, off);
      if ((lane & 7) == 0 && i < n) tile[q][i >> 3] = v;
    }
    __syncthreads();
    if (flags & 1) return false;
    if (warp < nq) {
      const int nt = (n + kCgrTile - 1) / kCgrTile;
      double v = 0.0;
      // (at most 96 tiles: three trees over 32, then 0 + 2 and that + 1, the
      // order of the tree over eight)
#pragma unroll 1
      for (int i = 0; i < 3; ++i) {
        const int j = i ? 3 - i : 0, m = nt - 32 * j;
        if (m <= 0) continue;
        double e = lane < m ? tile[warp][32 * j + lane] : 0.0;
#pragma unroll 1
        for (int off = 16; off > 0; off >>= 1)
          if (off < m) e += shfl_down(e, off);
        v = i ? v + e : e;
      }
      if (lane == 0) {
        tot[warp] = v;
        then(warp, v);
      }
    }
    __syncthreads();
    ++seq;
    return true;
  };

  __syncthreads();
  for (;;) {
    const bool first = it == 0;
    // ---- p = z + beta p: own rows, then the halo
    if (owner) {
      if (live) p = first ? z : fma(beta, p, z);
      vec[3 * mine + comp] = p;
    }
    bool ok = true;
    if (!first && B.nblk > 1) {
      ok = poll_recs<kHalo>(hv, [&](int j) { return A.pub + hc[j]; }, hw, ztag, err);
#pragma unroll
      for (int j = 0; j < kHalo; ++j)
        if (hw[j]) {
          double* q = vec + 3 * own + threadIdx.x + j * kThreads64;
          *q = fma(beta, *q, rec_double(hv[j]));
        }
      for (int i0 = 32 * warp + kHalo * kThreads64; i0 < 3 * B.nh; i0 += kThreads64) {
        const int i = i0 + lane;
        const bool want[1] = {i < 3 * B.nh};
        const uint4* src = A.pub + (want[0] ? 3 * (size_t)(B.row0 + __ldg(A.h_col + B.hoff + i / 3)) + i % 3 : 0);
        uint4 v[1] = {ld_rec(src)};
        ok = poll_recs<1>(v, [&](int) { return src; }, want, ztag, err) && ok;
        if (want[0]) {
          double* q = vec + 3 * own + i;
          *q = fma(beta, *q, rec_double(v[0]));
        }
      }
    }
    if (!__syncthreads_and(ok)) {
      cgr_abort(A, B);
      return;
    }
    // ---- Ap, (p, Ap)
    double a[4] = {0.0, 0.0, 0.0, 0.0};  // of part pt: slots k = j mod 4, j = pt (4 parts), 2 pt, 2 pt + 1 (2), all (1)
    if (roww) {
      const int per = 4 / parts;
#pragma unroll 1
      for (int j = 0; j < per; ++j) {
        const double* m = M.mat + 96 * comp + lane;
        double e = 0.0;
        int k = per * pt + j;
#pragma unroll 1
        for (; k < M.res; k += 4) {
          const double* u = vec + 3 * (int)M.li[32 * k + lane];
          e = fma(m[288 * k + 64], u[2], fma(m[288 * k + 32], u[1], fma(m[288 * k], u[0], e)));
        }
#pragma unroll 1
        for (; k < M.len; k += 4) {
          const double* u = vec + 3 * (int)M.gli[32 * k + lane];
          const double m0 = M.gell[ell_entry(M.soff, k, lane, 3 * comp)],
                       m1 = M.gell[ell_entry(M.soff, k, lane, 3 * comp + 1)],
                       m2 = M.gell[ell_entry(M.soff, k, lane, 3 * comp + 2)];
          e = fma(m2, u[2], fma(m1, u[1], fma(m0, u[0], e)));
        }
        a[0] = j == 0 ? e : a[0];
        a[1] = j == 1 ? e : a[1];
        a[2] = j == 2 ? e : a[2];
        a[3] = j == 3 ? e : a[3];
      }
      if (parts == 4) {
        if (pt > 0) sums[96 * B.nsl * (pt - 1) + ex_at] = a[0];
      } else if (parts == 2 && pt == 1) {
        sums[ex_at] = a[0] + a[1];
      }
    }
    __syncthreads();
    if (owner) {
      if (parts == 4)
        y = (a[0] + sums[ex_at]) + (sums[96 * B.nsl + ex_at] + sums[192 * B.nsl + ex_at]);
      else
        y = (a[0] + a[1]) + (parts == 2 ? sums[ex_at] : a[2] + a[3]);
      if (!live) y = 0.0;  // a row past the scene's adds nothing, whatever p holds
      ex[ex_at] = y;
    }
    __syncthreads();
    if (owner && comp == 0) {
      const double* q = ex + 96 * sl + lane;
      const double* u = vec + 3 * mine;
      slice_sum(0, fma(u[2], q[64], fma(u[1], q[32], u[0] * q[0])));
    }
    if (!total(1, [&]() { if (lane == 0) rcp = 1.0 / rz; }, [&](int, double v) { step[0] = rz / v; })) {
      cgr_abort(A, B);
      return;
    }
    alpha = step[0];
    // ---- x, r, z, (r, r), (r, z)
    if (owner) {
      if (live) {
        x = fma(alpha, p, x);
        r = fma(-alpha, y, r);
      }
      ex[ex_at] = r;
    }
    if (block_jacobi) {
      __syncthreads();
      if (owner) {
        const double* q = ex + 96 * sl + lane;
        z = fma(dv[2], q[64], fma(dv[1], q[32], dv[0] * q[0]));
      }
    } else {
      z = dv[0] * r;
    }
    if (owner) ex[96 * B.nsl + ex_at] = z;
    if (live && B.nblk > 1) st_rec(A.pub + 3 * (size_t)(B.row0 + row) + comp, rec_of(z, seq));
    __syncthreads();
    if (owner && comp < 2) {
      const double* q = ex + 96 * sl + lane;
      const double* o = q + (comp == 1 ? 96 * B.nsl : 0);
      slice_sum(comp, fma(q[64], o[64], fma(q[32], o[32], q[0] * o[0])));
    }
    ztag = seq;
    if (!total(2, []() {}, [&](int q, double v) { if (q == 1) step[1] = quotient_by(v, rz, rcp); })) {
      cgr_abort(A, B);
      return;
    }
    if (B.nblk > 1) halo_ahead();
    rr = tot[0];
    const unsigned long long bits = __double_as_longlong(rr);
    bool stop = false;
    if (bits < thr) {
      stop = true;
    } else {
      beta = step[1];
      rz_prev = rz;
      rz = tot[1];
      it = it + 1;
      if (it >= max_cg) {
        stop = true;
        cg_status = 5;  // MFEM_ERR_CG_MAXITER
      }
    }
    if ((bits & ~(1ull << 63)) > kInf) {  // NaN
      stop = true;
      status = 4;
    }
    if (stop) break;
  }
  // ---- the solution and the scene's scalars
  if (live) static_cast<double*>(sd.cg_x)[k4 + comp] = x;
  if (B.rec == 0 && threadIdx.x == 0) {
    sc_put(&sc->alpha, alpha);
    sc_put(&sc->beta, beta);
    sc_put(&sc->rz, rz);
    sc_put(&sc->rz_prev, rz_prev);
    sc->cg_err = cg_rel(rr, rr0);
    sc->cg_iter = it;
    sc->cg_total += it;
    if (status) sc->status = status;
    if (cg_status) sc->cg_status = cg_status;
    sc->cg_active = 0;
    sc->nph = kPhLocal;
    atomicSub(&A.ctrs->cg_active, 1);
    A.seq[B.scene] = seq;
  }
}

// --------------------------------------------- single-reduction form ---
// The mixed path's Chronopoulos-Gear iteration as cgf_tile runs it, from the
// state of the vectors of the current parity to the state after the last
// iteration done: until the recursion's stop is to be verified (cgf_phase set:
// the next launches of k_cgf_iter verify), or max_iters iterations.  The
// exchanged vector is w; each block keeps r and s at its halo.
struct CgfScalars {
  df64 gamma, alphaE, betaE, rr0, rr;
  df_rcp rg, ra;  // of gamma and alphaE
  float2 thr;
  float a, b;
  int it, rounds, phase, status, cg_status;
  bool swapped;  // an iteration left the recursion without counting (phase set)

  __device__ __forceinline__ explicit CgfScalars(const SceneScalars* sc)
      : gamma(sc_get<df64>(&sc->cgf_gamma[0])), alphaE(sc_get<df64>(&sc->alpha)), betaE(sc_get<df64>(&sc->beta)),
        rr0(sc_get<df64>(&sc->cg_rhs_norm2)), rr(rr0), thr(sc->cg_thr), a(sc->alpha_f), b(sc->beta_f), it(sc->cg_iter),
        rounds(sc->cgf_rounds), phase(0), status(0), cg_status(0), swapped(false) {}
  // While the sums travel.
  __device__ __forceinline__ void prepare() {
    rg = rcp_of(gamma);
    ra = rcp_of(alphaE);
  }
  // After an iteration's sums, as cgf_verify_step in phase 0: whether the launch ends.
  __device__ __forceinline__ bool step(const SceneDev& sd, const df64 (&d)[3]) {
    return advance(sd, d, [&](df64 g, df64* b, df64* ga) {
      *b = by_rcp(g, gamma, rg);
      *ga = by_rcp(g, alphaE, ra);
    });
  }
  // The same by a whole warp, whose even lanes take the quotients by gamma and
  // whose odd ones those by alpha, in the time of one.
  __device__ __forceinline__ df64 den() const { return threadIdx.x & 1 ? alphaE : gamma; }
  __device__ __forceinline__ void prepare_warp() { rg = rcp_of(den()); }
  __device__ __forceinline__ bool step_warp(const SceneDev& sd, const df64 (&d)[3]) {
    return advance(sd, d, [&](df64 g, df64* b, df64* ga) {
      const df64 v = by_rcp(g, den(), rg);
      *b = shfl_to(v, 0);
      *ga = shfl_to(v, 1);
    });
  }
  template <typename F>
  __device__ __forceinline__ bool advance(const SceneDev& sd, const df64 (&d)[3], const F& quotients) {
    rr = d[0];
    if (is_nan(rr)) {
      status = 4;
      phase = 3;
    } else if (cg_meets(sd, thr, rr, rr0)) {
      phase = rounds < kCgfRounds ? 1 : 3;
    }
    if (phase) {
      swapped = true;
      return true;
    }
    df64 ga;
    quotients(d[1], &betaE, &ga);
    alphaE = cgf_alpha(d[1], d[2], betaE, ga);
    gamma = d[1];
    a = to_step(alphaE);
    b = to_step(betaE);
    it += 1;
    if (it >= sd.max_cg) {
      cg_status = 5;  // MFEM_ERR_CG_MAXITER
      phase = 3;
      return true;
    }
    return false;
  }
  // the last iteration done
  __device__ __forceinline__ int last() const { return swapped ? it : it - 1; }
  __device__ __forceinline__ void store(SceneScalars* sc) const {
    sc->cg_err = cg_rel(rr, rr0);
    sc_put(&sc->beta, betaE);
    sc->beta_f = b;
    sc_put(&sc->alpha, alphaE);
    sc->alpha_f = a;
    sc_put(&sc->cgf_gamma[0], gamma);
    sc->cg_iter = it;
    sc->cgf_phase = phase;
    if (status) sc->status = status;
    if (cg_status) sc->cg_status = cg_status;
  }
};

template <bool kScaled, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) k_cgr_fused(const CgrArgs A) {
  extern __shared__ __align__(16) unsigned char cgr_smem_raw[];
  __shared__ CgrShared S;
  // The sums and the scalars, some 800 instructions an iteration, are warp 0's;
  // the others wait for the halo meanwhile.  (Every warp for itself: three
  // steps of 16 scenes in blocks of two tiles 27.0 ms, against 19.7, of six
  // scenes in blocks of one 14.4 against 13.8.)
  __shared__ float steps[2];  // warp 0's alpha and beta for the others
  __shared__ int leave, done;
  const CgrBlock B = A.blocks[blockIdx.x];
  const SceneDev& sd = A.sds[B.scene];
  SceneScalars* sc = sd.sc;
  if (!sc->cg_active || sc->cgf_phase) return;
  unsigned seq = __ldcg(A.seq + B.scene);
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  if (threadIdx.x == 0) S.late = 0;
  CgfScalars q(sc);
  const bool roww = sl < B.nsl;
  const int row = 32 * (B.slice0 + sl) + lane;
  const bool live = roww && row < sd.nf;
  const int own = 32 * B.nsl, mine = 32 * sl + lane;
  unsigned char* rest;
  const CgrMatrix<float> M = cgr_load_matrix<float>(A, B, sd, sl, cgr_smem_raw, &rest);
  float4* u4 = reinterpret_cast<float4*>(rest);         // u at the own rows and the halo
  float4* sh = u4 + own + B.nh;                         // s at the halo
  float4* rh = kScaled ? u4 + own : sh + B.nh;          // r at the halo (scaled: u itself)
  float* Dh = reinterpret_cast<float*>(sh + 2 * B.nh);  // unscaled: M^-1 at the halo, 9 each
  const int it = q.it;
  const float* gr = static_cast<const float*>(sd.cgf_r[it & 1]);
  const float* gw = static_cast<const float*>(sd.cgf_w[it & 1]);
  const float* gs = static_cast<const float*>(sd.cgf_s[(it + 1) & 1]);
  int hc[kHaloRegs];
  bool hw[kHaloRegs];
  uint4 hv[kHaloRegs];
#pragma unroll
  for (int j = 0; j < kHaloRegs; ++j) {
    const int h = threadIdx.x + j * kThreads;
    hw[j] = h < B.nh;
    hc[j] = hw[j] ? A.h_col[B.hoff + h] : 0;
    if (hw[j]) hv[j] = *reinterpret_cast<const uint4*>(gw + 4 * (size_t)hc[j]);
  }
  for (int h = threadIdx.x; h < B.nh; h += kThreads) {
    const int col = A.h_col[B.hoff + h];
    rh[h] = *reinterpret_cast<const float4*>(gr + 4 * (size_t)col);
    sh[h] = *reinterpret_cast<const float4*>(gs + 4 * (size_t)col);
    if (!kScaled) {
      const float* dinv = static_cast<const float*>(sd.dinv);
      if (sd.block_jacobi) {
        for (int c = 0; c < 9; ++c) Dh[9 * h + c] = dinv[9 * (size_t)col + c];
      } else {
        for (int c = 0; c < 3; ++c) Dh[9 * h + c] = dinv[4 * (size_t)col + c];
      }
    }
  }
  const size_t k4 = 4 * (size_t)row;
  float r[3] = {0.f, 0.f, 0.f}, w[3] = {0.f, 0.f, 0.f}, s[3] = {0.f, 0.f, 0.f}, p[3] = {0.f, 0.f, 0.f},
        x[3] = {0.f, 0.f, 0.f}, u[3] = {0.f, 0.f, 0.f}, dv[3] = {1.f, 1.f, 1.f};
  if (live) {
    ld3<false>(gr + k4, r);
    ld3<false>(gw + k4, w);
    ld3<false>(gs + k4, s);
    ld3<false>(static_cast<const float*>(sd.cg_p[0]) + k4, p);
    ld3<false>(static_cast<const float*>(sd.cg_x) + k4, x);
    if (kScaled) ld3<false>(static_cast<const float*>(sd.dinv) + k4, dv);
    else ld3<false>(static_cast<const float*>(sd.cg_z) + k4, u);
  }
  unsigned wtag = 0;

  for (int n = 0;; ++n) {
    const bool first = n == 0;
    const float a = q.a, b = q.b;
    // ---- own rows: s, r, u, p, x of iteration it + 1
    float rn[3], un[3];
    if (live) {
      float sv[3], uv[3];
      if (kScaled) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          sv[c] = fma(b, s[c], w[c]);
          un[c] = fma(-a, sv[c], r[c]);
          rn[c] = un[c] / dv[c];
          uv[c] = r[c];
        }
      } else {
        cgf_next<float>(sd, row, r, w, s, a, b, sv, rn, un);
#pragma unroll
        for (int c = 0; c < 3; ++c) uv[c] = u[c];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        p[c] = fma(b, p[c], uv[c]);
        x[c] = fma(a, p[c], x[c]);
        s[c] = sv[c];
        r[c] = kScaled ? un[c] : rn[c];
        u[c] = un[c];
      }
      u4[mine] = make_float4(un[0], un[1], un[2], 0.f);
    } else if (roww) {
      u4[mine] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // ---- the halo's s, r and u
    const uint4* pw = A.pub + (size_t)(wtag & 1) * A.pub_stride + B.row0;
    bool ok = true;
    auto halo = [&](int h, const uint4& v) {
      const float wc[3] = {__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z)};
      const float4 so = sh[h], ro = rh[h];
      const float sn[3] = {fma(b, so.x, wc[0]), fma(b, so.y, wc[1]), fma(b, so.z, wc[2])};
      const float rc[3] = {fma(-a, sn[0], ro.x), fma(-a, sn[1], ro.y), fma(-a, sn[2], ro.z)};
      sh[h] = make_float4(sn[0], sn[1], sn[2], 0.f);
      rh[h] = make_float4(rc[0], rc[1], rc[2], 0.f);
      if (!kScaled) {
        float uc[3];
        const float* D = Dh + 9 * h;
        if (sd.block_jacobi) {
#pragma unroll
          for (int c = 0; c < 3; ++c) uc[c] = fma(D[3 * c + 2], rc[2], fma(D[3 * c + 1], rc[1], D[3 * c] * rc[0]));
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) uc[c] = D[c] * rc[c];
        }
        u4[own + h] = make_float4(uc[0], uc[1], uc[2], 0.f);
      }
    };
    if (!first) ok = poll_recs<kHaloRegs>(hv, [&](int j) { return pw + hc[j]; }, hw, wtag, &A.ctrs->error) && ok;
#pragma unroll
    for (int j = 0; j < kHaloRegs; ++j)
      if (hw[j]) halo(threadIdx.x + j * kThreads, hv[j]);
    for (int h0 = 32 * sl + kHaloRegs * kThreads; h0 < B.nh; h0 += kThreads) {
      const int h = h0 + lane;
      const bool want[1] = {h < B.nh};
      const int col = want[0] ? __ldg(A.h_col + B.hoff + h) : 0;
      const uint4* src = first ? reinterpret_cast<const uint4*>(gw + 4 * (size_t)col) : pw + col;
      uint4 v[1] = {ld_rec(src)};
      if (!first) ok = poll_recs<1>(v, [&](int) { return src; }, want, wtag, &A.ctrs->error) && ok;
      if (want[0]) halo(h, v[0]);
    }
    if (!__syncthreads_and(ok)) {
      cgr_abort(A, B);
      return;
    }
    // ---- w = A u, (r, r), (r, u), (w, u)
    df64 d[3] = {df64(0.f), df64(0.f), df64(0.f)};
    if (roww) {
      float acc[3] = {0.f, 0.f, 0.f};
      cgr_multiply(M, u4, acc);
#pragma unroll
      for (int c = 0; c < 3; ++c) w[c] = kScaled ? dv[c] * acc[c] : acc[c];
      if (live) {
        if (B.nblk > 1)
          st_rec(A.pub + (size_t)(seq & 1) * A.pub_stride + B.row0 + row,
                 make_uint4(__float_as_uint(w[0]), __float_as_uint(w[1]), __float_as_uint(w[2]), seq));
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          d[0] = acc_prod(d[0], rn[c], rn[c]);
          d[1] = acc_prod(d[1], rn[c], un[c]);
          d[2] = acc_prod(d[2], acc[c], un[c]);
        }
      }
    }
    bool got = scene_total<df64, 3, true>(A, B, S, roww, sl, seq, d, [&]() {
#pragma unroll
          for (int j = 0; j < kHaloRegs; ++j)
            if (hw[j]) hv[j] = ld_rec(A.pub + (size_t)(seq & 1) * A.pub_stride + B.row0 + hc[j]);
        }, [&]() { if (sl == 0) q.prepare_warp(); });
    wtag = seq;
    ++seq;
    if (sl > 0)
      got = poll_recs<kHaloRegs>(hv, [&](int j) { return A.pub + (size_t)(wtag & 1) * A.pub_stride + B.row0 + hc[j]; },
                                 hw, wtag, &A.ctrs->error) && got;
    if (got && sl == 0) {
      const bool stop = q.step_warp(sd, d) || n + 1 >= A.max_iters;
      if (lane == 0) {
        leave = stop;
        done = q.last();
        steps[0] = q.a;
        steps[1] = q.b;
      }
    }
    // (no warp goes on without warp 0, whose step ends the loop)
    if (!__syncthreads_and(got)) {
      cgr_abort(A, B);
      return;
    }
    if (leave) break;
    q.a = steps[0];
    q.b = steps[1];
  }
  const int last = done;
  // ---- the vectors as k_cgf_iter leaves them after iteration `last`
  if (live) {
    st3(static_cast<float*>(sd.cgf_r[(last + 1) & 1]) + k4, r);
    st3(static_cast<float*>(sd.cgf_w[(last + 1) & 1]) + k4, w);
    st3(static_cast<float*>(sd.cgf_s[last & 1]) + k4, s);
    st3(static_cast<float*>(sd.cg_p[0]) + k4, p);
    st3(static_cast<float*>(sd.cg_x) + k4, x);
    if (!kScaled) st3(static_cast<float*>(sd.cg_z) + k4, u);
  }
  if (B.rec == 0 && threadIdx.x == 0) {
    q.store(sc);
    A.seq[B.scene] = seq;
  }
}

// The same iteration for batches whose matrices outgrow the shared memory of
// all SMs (more than two tiles an SM; up to six).  A block is up to 48 slices,
// a warp up to three, with their rows' vectors in registers; the matrix streams
// through a ring of slots in shared memory, as in the staged k_cgf_iter, and
// little else leaves the SM: the rows' u, their x and the sums, where the launch
// per iteration reads three vectors at every neighbour and writes five.  The
// ring runs on from one iteration into the next, so that it is full when the
// sums of the last have come in.  The exchanged vector is u itself: the halo
// takes 20 bytes of shared memory a column, and the iteration waits twice, for
// the neighbours' rows and for the sums.
//
// (A later build, by events: 16.6 us at 85k rows, 26.4 at 223k.)
// An iteration at 85k / 130k / 148k / 223k rows: 17.9 / 21.3 / 21.6 / 32.0 us,
// against 25.4 / 28.1 / 30.2 / 37.9 us in launches (block Jacobi: 18.3 / 21.9 /
// 22.3 / 33.7 against 32.3 / 35.3 / 37.0 / 50.9).  Of the 62,000 cycles at 223k
// rows the product is 30,000 (128 MB, 19 us of DRAM time, of which the L2 keeps
// a quarter; a slot passes shared memory twice, 20,000 cycles), the own rows
// 6,500, the halo 3,500, waiting for the slowest warp and block and the sums
// the rest.  One slot at a time with its refill: 38,000 cycles for the product;
// neighbouring slices in a warp, of unlike lengths: 36,000; the matrix in
// registers from plain loads with a fifth of it resident: 62,000.  Prefetching
// the next iteration's slots to L2 while the sums travel slowed the sums by
// what it saved.
constexpr int kCgrTake = 2;  // slots out of the ring at a time
constexpr int kWideWarps = kCgrWideWarps, kWideThreads = 32 * kWideWarps, kWideSlices = kCgrWideSlices / kWideWarps;

// `tree` over 32 lanes for N values at once: each level leaves one half of the
// lanes one value of a pair and the other half the other, so that N values
// take about N + 5 additions in place of 5 N.  (The pairs added are the
// tree's, and an addition's operands may change places.)  Afterwards lane l
// holds the value of index *i.
template <int N, int kOff = 16>
__device__ __forceinline__ df64 trees(const df64 (&v)[N], int* i) {
  const int lane = threadIdx.x & 31;
  const bool up = (lane & kOff) != 0;
  constexpr int M = (N + 1) / 2;
  df64 a[M];
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const df64 lo = v[2 * j], hi = v[2 * j + 1 < N ? 2 * j + 1 : 2 * j];
    const df64 keep = up ? hi : lo, send = up ? lo : hi;
    a[j] = keep + df64(__shfl_xor_sync(0xffffffffu, send.hi, kOff), __shfl_xor_sync(0xffffffffu, send.lo, kOff));
  }
  if constexpr (kOff > 1) {
    const df64 t = trees<M, kOff / 2>(a, i);
    *i = min(2 * *i + (up ? 1 : 0), N - 1);
    return t;
  } else {
    static_assert(M == 1, "at most 32 values");
    *i = min(up ? 1 : 0, N - 1);
    return a[0];
  }
}

template <bool kScaled>
__global__ void __launch_bounds__(kWideThreads, 1) k_cgr_wide(const CgrArgs A) {
  extern __shared__ __align__(16) unsigned char cgr_smem_raw[];
  __shared__ double part[3][kCgrWideSlices], red[3][8];
  __shared__ int lens[kCgrWideSlices], offs[kCgrWideSlices], who[kCgrWideSlices];  // of the slices in the warps' order
  __shared__ __align__(8) unsigned char q_raw[sizeof(CgfScalars)];
  CgfScalars& q = *reinterpret_cast<CgfScalars*>(q_raw);
  __shared__ int leave;
  constexpr int kHalo = 4;
  const CgrBlock B = A.blocks[blockIdx.x];
  const SceneDev& sd = A.sds[B.scene];
  SceneScalars* sc = sd.sc;
  if (!sc->cg_active || sc->cgf_phase) return;
  unsigned seq = __ldcg(A.seq + B.scene);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* err = &A.ctrs->error;

  // ---- the warp's slices (B.pick: of like numbers of slots in all warps) and
  // its ring: S stages of a slot's 160 pairs and 32 local column indices, one
  // mbarrier each; the slots of the slices one after another, over and over
  const int first = kWideSlices * warp;
  int sl[kWideSlices], nslots = 0, ns = 0;
  const int soff0 = sd.slice_off[B.slice0];
#pragma unroll
  for (int j = 0; j < kWideSlices; ++j) {
    sl[j] = B.pick[first + j];
    if (sl[j] < B.nsl) {
      const int off = sd.slice_off[B.slice0 + sl[j]], len = (sd.slice_off[B.slice0 + sl[j] + 1] - off) >> 5;
      nslots += len;
      ns = j + 1;
      if (lane == 0) {
        lens[first + j] = len;
        offs[first + j] = off;
        who[first + j] = sl[j];
      }
    }
  }
  __syncwarp();
  const int own = 32 * B.nsl;
  float4* u4 = reinterpret_cast<float4*>(cgr_smem_raw);  // u at the own rows and the halo
  int* hcol = reinterpret_cast<int*>(u4 + own + B.nh);  // the halo's columns
  for (int h = threadIdx.x; h < B.nh; h += kWideThreads) hcol[h] = A.h_col[B.hoff + h];
  const uint32_t ring = smem_addr(hcol + (B.nh + 3) / 4 * 4);
  const uint32_t bar0 = ring + 8u * (uint32_t)(warp * B.kres);
  const uint32_t stage0 = ring + 8u * (uint32_t)(kWideWarps * B.kres) +
                          kCgrStage * (uint32_t)(warp * B.kres);
  const float2* ell = static_cast<const float2*>(sd.ell);
  const uint16_t* gli = A.lidx + B.loff;
  const int S = min(B.kres, nslots);
  // the slot the next fill fetches (lane 0): slice, slots left of it, addresses
  int fj = -1, frem = 0;
  const float2* fe = ell;
  const uint16_t* fl = gli;
  const unsigned long long pol = l2_matrix_policy<2>();
  auto to_next = [&]() {
    fj = fj + 1 == ns ? 0 : fj + 1;
    frem = lens[first + fj];
    fe = ell + 5 * (size_t)offs[first + fj];
    fl = gli + (offs[first + fj] - soff0);
  };
  auto fill = [&](int stage) {
    const uint32_t bar = bar0 + 8u * stage, dst = stage0 + kCgrStage * stage;
    mbar_arrive_expect_tx(bar, kCgrStage);
    bulk_g2s(dst, fe, 1280u, bar, pol);
    bulk_g2s(dst + 1280u, fl, 64u, bar, pol);
    fe += 160;
    fl += 32;
    if (--frem == 0) to_next();
  };
  if (lane == 0)
    for (int i = 0; i < S; ++i) mbar_init(bar0 + 8u * i, 1u);
  fence_mbar_init();
  __syncwarp();
  if (lane == 0 && S > 0) {
    to_next();
    for (int i = 0; i < S; ++i) fill(i);
  }
  int st = 0;          // the stage read next
  uint32_t round = 0;  // its parity
  // every copy in flight lands before the block leaves (S of them, always)
  auto drain = [&]() {
    for (int i = 0; i < S; ++i) {
      mbar_wait(bar0 + 8u * st, round);
      st = st + 1 == S ? 0 : st + 1;
      round ^= st == 0;
    }
    __syncwarp();
  };

  // ---- the rows' vectors
  if (threadIdx.x == 0) new (&q) CgfScalars(sc);
  const int it = sc->cg_iter;
  const float* gr = static_cast<const float*>(sd.cgf_r[it & 1]);
  const float* gw = static_cast<const float*>(sd.cgf_w[it & 1]);
  const float* gs = static_cast<const float*>(sd.cgf_s[(it + 1) & 1]);
  // (u, which is the scaled r, stays in u4); dr: M^-1 (scaled) or r
  float w[kWideSlices][3], sv[kWideSlices][3], p[kWideSlices][3], dr[kWideSlices][3];
  float* gx = static_cast<float*>(sd.cg_x);  // x: read and written once an iteration, off the chain
  bool live[kWideSlices];
#pragma unroll
  for (int j = 0; j < kWideSlices; ++j) {
    const int row = 32 * (B.slice0 + sl[j]) + lane;
    live[j] = j < ns && row < sd.nf;
#pragma unroll
    for (int c = 0; c < 3; ++c) w[j][c] = sv[j][c] = p[j][c] = dr[j][c] = 0.f;
    if (live[j]) {
      const size_t k4 = 4 * (size_t)row;
      ld3<false>(gw + k4, w[j]);
      ld3<false>(gs + k4, sv[j]);
      ld3<false>(static_cast<const float*>(sd.cg_p[0]) + k4, p[j]);
      float u[3];
      ld3<false>(kScaled ? static_cast<const float*>(sd.dinv) + k4 : gr + k4, dr[j]);
      ld3<false>(kScaled ? gr + k4 : static_cast<const float*>(sd.cg_z) + k4, u);
      u4[32 * sl[j] + lane] = make_float4(u[0], u[1], u[2], 0.f);
    }
  }
  uint4* pub = A.pub + B.row0;
  const int copies = exchange_copies(B.nblk);
  const size_t cstride = 3 * (size_t)A.nrec_total;
  __syncthreads();

  for (int n = 0;; ++n) {
    const float a = q.a, b = q.b;
    // ---- own rows: s, r, u, p, x of iteration it + 1; (r, r), (r, u)
    {
      df64 e[2 * kWideSlices];
#pragma unroll
      for (int j = 0; j < kWideSlices; ++j) {
        const int row = 32 * (B.slice0 + sl[j]) + lane;
        float un[3] = {0.f, 0.f, 0.f};
        e[2 * j] = e[2 * j + 1] = df64(0.f);
        if (live[j]) {
          float rn[3], sn[3];
          const float4 u = u4[32 * sl[j] + lane];
          const float uv[3] = {u.x, u.y, u.z};
          if (kScaled) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              sn[c] = fma(b, sv[j][c], w[j][c]);
              un[c] = fma(-a, sn[c], uv[c]);
              rn[c] = un[c] / dr[j][c];
            }
          } else {
            cgf_next<float>(sd, row, dr[j], w[j], sv[j], a, b, sn, rn, un);
          }
          if (B.nblk > 1)
            st_rec(pub + row,
                   make_uint4(__float_as_uint(un[0]), __float_as_uint(un[1]), __float_as_uint(un[2]), seq));
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            p[j][c] = fma(b, p[j][c], uv[c]);
            sv[j][c] = sn[c];
            if (!kScaled) dr[j][c] = rn[c];
            e[2 * j] = acc_prod(e[2 * j], rn[c], rn[c]);
            e[2 * j + 1] = acc_prod(e[2 * j + 1], rn[c], un[c]);
          }
        }
        if (j < ns) u4[32 * sl[j] + lane] = make_float4(un[0], un[1], un[2], 0.f);
      }
      int i;
      const df64 t = trees(e, &i);
      if ((i >> 1) < ns) Slot<df64>::put(&part[i & 1][who[first + (i >> 1)]], t);
    }
    // ---- the halo's u
    bool ok = true;
    for (int h0 = 32 * warp; h0 < B.nh; h0 += kHalo * kWideThreads) {
      uint4 v[kHalo];
      bool want[kHalo];
      int col[kHalo];
#pragma unroll
      for (int j = 0; j < kHalo; ++j) {
        const int h = h0 + j * kWideThreads + lane;
        want[j] = h < B.nh;
        col[j] = want[j] ? hcol[h] : 0;
      }
#pragma unroll
      for (int j = 0; j < kHalo; ++j)
        if (want[j]) v[j] = ld_rec(pub + col[j]);
      ok = poll_recs<kHalo>(v, [&](int j) { return pub + col[j]; }, want, seq, err) && ok;
#pragma unroll
      for (int j = 0; j < kHalo; ++j)
        if (want[j])
          u4[own + h0 + j * kWideThreads + lane] =
              make_float4(__uint_as_float(v[j].x), __uint_as_float(v[j].y), __uint_as_float(v[j].z), 0.f);
    }
    if (!__syncthreads_and(ok)) {
      drain();
      cgr_abort(A, B);
      return;
    }
    // ---- w = A u, (w, u)
    float aw[kWideSlices][3];
#pragma unroll 1
    for (int j = 0; j < ns && ok; ++j) {
      float acc[3] = {0.f, 0.f, 0.f};
      const int len = lens[first + j];
      // n slots: out of their stages, the stages refilled, the products
      auto take = [&](auto n_) -> bool {
        constexpr int n = decltype(n_)::value;
        int at[n];
        bool got = true;
#pragma unroll
        for (int i = 0; i < n; ++i) {
          at[i] = st;
          got = mbar_wait(bar0 + 8u * st, round) && got;
          st = st + 1 == S ? 0 : st + 1;
          round ^= st == 0;
        }
        if (!__all_sync(0xffffffffu, got)) return false;
        float2 e[n][5];
        unsigned short col[n];
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const uint32_t src = stage0 + kCgrStage * at[i];
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(col[i]) : "r"(src + 1280u + 2u * lane) : "memory");
#pragma unroll
          for (int c = 0; c < 5; ++c) e[i][c] = lds_pair(src + 256u * c + 8u * lane, 0.f);
        }
        __syncwarp();
        if (lane == 0) {
          fence_proxy_async_smem();
#pragma unroll
          for (int i = 0; i < n; ++i) fill(at[i]);
        }
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const float4 t = u4[col[i]];
          const float uc[3] = {t.x, t.y, t.z};
          ell_block_fma(e[i][0], e[i][1], e[i][2], e[i][3], e[i][4], uc, acc[0], acc[1], acc[2]);
        }
        return true;
      };
      int k = 0;
#pragma unroll 1
      for (; ok && k + kCgrTake <= len; k += kCgrTake) ok = take(std::integral_constant<int, kCgrTake>());
#pragma unroll 1
      for (; ok && k < len; ++k) ok = take(std::integral_constant<int, 1>());
#pragma unroll
      for (int i = 0; i < kWideSlices; ++i)
        if (i == j)
#pragma unroll
          for (int c = 0; c < 3; ++c) aw[i][c] = acc[c];
    }
    if (!ok && lane == 0) atomicExch(err, 1);
    {
      df64 e[kWideSlices];
#pragma unroll
      for (int j = 0; j < kWideSlices; ++j) {
        e[j] = df64(0.f);
        if (live[j]) {
          const float4 t = u4[32 * sl[j] + lane];
          const float u[3] = {t.x, t.y, t.z};
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            w[j][c] = kScaled ? dr[j][c] * aw[j][c] : aw[j][c];
            e[j] = acc_prod(e[j], aw[j][c], u[c]);
          }
        }
      }
      int i;
      const df64 t = trees(e, &i);
      if (i < ns) Slot<df64>::put(&part[2][who[first + i]], t);
    }
    if (!__syncthreads_and(ok)) {
      drain();
      cgr_abort(A, B);
      return;
    }
    // ---- the tiles' sums to every block: lane 8 t + c sends copy c of tile t
    {
      uint4* rec = A.recs + (seq & 1) * kMaxCopies * cstride + B.rec0 + B.rec;
      const int groups = (B.nsl + 31) / 32;
      for (int job = warp; job < 3 * groups; job += kWideWarps) {
        const int i = job / groups, s = 32 * (job % groups) + lane;
        df64 v[1] = {s < B.nsl ? Slot<df64>::sget(&part[i][s]) : df64(0.f)};
        tree<df64, 1, 4>(v);
        const df64 t(__shfl_sync(0xffffffffu, v[0].hi, lane & 24), __shfl_sync(0xffffffffu, v[0].lo, lane & 24));
        if ((lane & 7) < copies && (s & ~7) < B.nsl)
          st_rec(rec + (lane & 7) * cstride + (size_t)i * A.nrec_total + (s >> 3), rec_of(t, seq));
      }
    }
    // ---- x, while the sums travel
    if (threadIdx.x == 0) q.prepare();
#pragma unroll
    for (int j = 0; j < kWideSlices; ++j)
      if (live[j]) {
        float x[3];
        float* at = gx + 4 * (size_t)(32 * (B.slice0 + sl[j]) + lane);
        ld3<false>(at, x);
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c] = fma(a, p[j][c], x[c]);
        st3(at, x);
      }
    // ---- all sums, in the order of scene_sums (a thread the tiles i, i + 256,
    // ..): eight warps a sum, the third one's the first eight's second
    {
      const int g = warp & 7, first = 32 * g + lane;
      const uint4* src = A.recs + ((seq & 1) * kMaxCopies + blockIdx.x % copies) * cstride + B.rec0 + first;
#pragma unroll 1
      for (int i = warp >> 3; i < 3; i += 2) {
        const uint4* at = src + i * (size_t)A.nrec_total;
        uint4 v[4];
        bool want[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          want[j] = first + 256 * j < B.nrec;
          if (want[j]) v[j] = ld_rec(at + 256 * j);
        }
        ok = poll_recs<4>(v, [&](int j) { return at + 256 * j; }, want, seq, err) && ok;
        df64 e[1] = {df64(0.f)};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (want[j]) e[0] = e[0] + rec_val<df64>(v[j]);
        tree<df64, 1, 16>(e);
        if (lane == 0) Slot<df64>::put(&red[i][g], e[0]);
      }
    }
    if (!__syncthreads_and(ok)) {
      drain();
      cgr_abort(A, B);
      return;
    }
    if (warp == 0) {
      df64 d[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) d[i] = lane < 8 ? Slot<df64>::sget(&red[i][lane]) : df64(0.f);
      tree<df64, 3, 4>(d);
      if (lane == 0) leave = q.step(sd, d) || n + 1 >= A.max_iters;
    }
    __syncthreads();
    ++seq;
    if (leave) break;
  }
  drain();
  // ---- the vectors as k_cgf_iter leaves them after iteration `last`
  const int last = q.last();
#pragma unroll
  for (int j = 0; j < kWideSlices; ++j)
    if (live[j]) {
      const size_t k4 = 4 * (size_t)(32 * (B.slice0 + sl[j]) + lane);
      const float4 t = u4[32 * sl[j] + lane];
      const float u[3] = {t.x, t.y, t.z};
      if (kScaled) {
        st3(static_cast<float*>(sd.cgf_r[(last + 1) & 1]) + k4, u);
      } else {
        st3(static_cast<float*>(sd.cgf_r[(last + 1) & 1]) + k4, dr[j]);
        st3(static_cast<float*>(sd.cg_z) + k4, u);
      }
      st3(static_cast<float*>(sd.cgf_w[(last + 1) & 1]) + k4, w[j]);
      st3(static_cast<float*>(sd.cgf_s[last & 1]) + k4, sv[j]);
      st3(static_cast<float*>(sd.cg_p[0]) + k4, p[j]);
    }
  if (B.rec == 0 && threadIdx.x == 0) {
    q.store(sc);
    A.seq[B.scene] = seq;
  }
}

template <typename F> auto with_kernel(bool fp64, bool fused, bool jacobi, bool wide, int threads, F&& f) {
  if (wide) return jacobi ? f((const void*)k_cgr_wide<true>) : f((const void*)k_cgr_wide<false>);
  if (fused && threads > 256) return jacobi ? f((const void*)k_cgr_fused<true, 512>) : f((const void*)k_cgr_fused<false, 512>);
  if (fused) return jacobi ? f((const void*)k_cgr_fused<true, 256>) : f((const void*)k_cgr_fused<false, 256>);
  if (fp64) return f((const void*)k_cgr_split64);
  return threads > 256 ? f((const void*)k_cgr_split<512>) : f((const void*)k_cgr_split<256>);
}

}  // namespace

int cgr_blocks_per_sm(bool fp64, bool fused, bool jacobi, bool wide, int threads, size_t smem) {
  return with_kernel(fp64, fused, jacobi, wide, threads, [&](const void* k) {
    int nb = 0;
    // the function's limit is shared by every batch: always the largest
    if (smem > kCgrSmem ||
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCgrSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, threads, smem) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return nb;
  });
}

cudaError_t launch_cgr(const CgrArgs& args, bool fp64, bool fused, bool jacobi, bool wide, int nblocks, int threads,
                       size_t smem, cudaStream_t stream) {
  return with_kernel(fp64, fused, jacobi, wide, threads, [&](const void* k) {
    CgrArgs a = args;
    void* params[] = {&a};
    return cudaLaunchCooperativeKernel(k, dim3(nblocks), dim3(threads), params, smem, stream);
  });
}

}  // namespace mfem_gpu
