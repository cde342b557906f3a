// Block-Jacobi PCG on a caller-owned, device-resident 3x3 block-CSR matrix
// that allocates nothing: every scratch vector, the tile partials, the
// tickets and the scalars live in one file-scope __device__ array of fixed
// size (MFEM_NOALLOC_PCG_MAX_ROWS block rows).
//
// Two forms of the same iteration.  k_na_resident runs the whole solve in one
// cooperative launch with the matrix in shared memory; it hands back a system
// that it does not fit (or whose pattern or diagonal is not in order) before
// it has changed anything, and the launches of k_na_init, k_na_spmv and
// k_na_update, two an iteration, then take it.
//
// The iteration is the one of the scene PCG (Eigen's ConjugateGradient with
// a block-diagonal preconditioner, src/linear_solvers/eigen_iterative_solver.h:20-29):
// x0 = 0, stop when |r|^2 < tol^2 |b|^2 or after max_iters iterations.  The
// p update is folded into the SpMV (p = z + beta p_prev formed per column),
// and the dot products are reduced deterministically: fixed-order block
// sums per tile, then the last tile (atomic ticket, no thread waits) sums
// the tile partials in tile order.
//
// Scratch state and what must start at zero: the ticket counter.  It is zero
// when the module loads, the last tile of every kernel returns it to zero,
// and each call clears the scalar block (ticket included) with
// cudaMemsetAsync before its first kernel.  Everything else in the scratch
// is written before it is read within a call.
//
// Calls on one device share that scratch, so two calls that overlapped on
// one device would race.  The entry point therefore holds that device's
// lock from its first launch until its stream has drained; calls on
// different devices use different scratch copies and different locks.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "../../include/mfem_gb300.h"
#include "exchange.cuh"

namespace {

constexpr int kNaThreads = 256;
constexpr int kNaMaxRows = MFEM_NOALLOC_PCG_MAX_ROWS;
constexpr int kNaMaxTiles = (kNaMaxRows + kNaThreads - 1) / kNaThreads;
constexpr int kNaChunk = 16;  // iterations launched between two host checks
constexpr int kNaMaxDevices = 64;

struct NaScalars {
  double rr0, thr, rz, alpha, beta, err;
  int iter, active, status, max_iters;
  unsigned int ticket;
  int done;   // k_na_resident: 1 solved (status, iter, err hold), 0 handed back
  int error;  // a wait of k_na_resident ran out
};

constexpr size_t na_align(size_t v) { return (v + 255) / 256 * 256; }
constexpr size_t kNaVecBytes = 3 * sizeof(double) * (size_t)kNaMaxRows;
constexpr size_t kNaOffPartials = na_align(sizeof(NaScalars));
constexpr size_t kNaOffDinv = na_align(kNaOffPartials + 2 * sizeof(double) * kNaMaxTiles);
constexpr size_t kNaOffVecs = na_align(kNaOffDinv + 9 * sizeof(double) * (size_t)kNaMaxRows);
// k_na_resident: its exchange's next tag, its blocks' tagged sums [parity][copy][2]
// and the tagged vector [3 n] (kept from call to call: their tags go on)
constexpr int kNaMaxBlocks = 160;
constexpr size_t kNaOffSeq = na_align(kNaOffVecs + 5 * kNaVecBytes);  // r, z, p0, p1, Ap
constexpr size_t kNaOffRecs = kNaOffSeq + 256;
constexpr size_t kNaOffPub = na_align(kNaOffRecs + 4 * mfem_gpu::kMaxCopies * sizeof(uint4) * kNaMaxBlocks);
constexpr size_t kNaScratchBytes = kNaOffPub + 3 * sizeof(uint4) * (size_t)kNaMaxRows;
static_assert(kNaScratchBytes < (size_t(8) << 20), "scratch stays a few MiB");

static __device__ __align__(256) unsigned char g_na_scratch[kNaScratchBytes];

struct NaView {
  NaScalars* sc;
  double* partials;  // [2][kNaMaxTiles]
  double* dinv;      // 9 per row, row-major 3x3
  double* r;
  double* z;
  double* p[2];
  double* Ap;
  unsigned int* seq;
  uint4* recs;
  uint4* pub;
};

NaView na_view(unsigned char* base) {
  NaView v;
  v.sc = reinterpret_cast<NaScalars*>(base);
  v.partials = reinterpret_cast<double*>(base + kNaOffPartials);
  v.dinv = reinterpret_cast<double*>(base + kNaOffDinv);
  double* vec = reinterpret_cast<double*>(base + kNaOffVecs);
  const size_t n3 = 3 * (size_t)kNaMaxRows;
  v.r = vec;
  v.z = vec + n3;
  v.p[0] = vec + 2 * n3;
  v.p[1] = vec + 3 * n3;
  v.Ap = vec + 4 * n3;
  v.seq = reinterpret_cast<unsigned int*>(base + kNaOffSeq);
  v.recs = reinterpret_cast<uint4*>(base + kNaOffRecs);
  v.pub = reinterpret_cast<uint4*>(base + kNaOffPub);
  return v;
}

struct NaMatrix {
  int n, nnzb;
  const int32_t* row_ptr;
  const int32_t* col;
  const double* val;
};

// Fixed-order block sums of NQ values; written as tile partials by thread 0.
template <int NQ>
__device__ __forceinline__ void na_tile_partials(double (&v)[NQ], double* partials) {
  __shared__ double red[kNaThreads / 32][NQ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], off);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) red[warp][q] = v[q];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double a = red[0][q];
      for (int w = 1; w < kNaThreads / 32; ++w) a += red[w][q];
      partials[q * kNaMaxTiles + blockIdx.x] = a;
    }
}

// True in thread 0 of the tile that arrived last; that thread then sees
// every other tile's partials.
__device__ __forceinline__ bool na_last_tile(NaScalars* sc) {
  if (threadIdx.x != 0) return false;
  __threadfence();
  if (atomicAdd(&sc->ticket, 1u) + 1u != gridDim.x) return false;
  sc->ticket = 0u;
  __threadfence();
  return true;
}

// Status flags raised by atomics of other tiles in the same launch.
__device__ __forceinline__ int na_status(NaScalars* sc) { return *(volatile int*)&sc->status; }

__device__ __forceinline__ double na_sum(const double* partials, int q) {
  double a = 0.0;
  for (int t = 0; t < (int)gridDim.x; ++t) a += __ldcg(partials + q * kNaMaxTiles + t);
  return a;
}

__device__ __forceinline__ void na_prec(const double* D, const double r[3], double z[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) z[c] = D[3 * c] * r[0] + D[3 * c + 1] * r[1] + D[3 * c + 2] * r[2];
}

// True if the row's entries lie inside the matrix; records MFEM_ERR_INVALID
// otherwise, so that a malformed pattern is skipped instead of read.
__device__ __forceinline__ bool na_row_ok(const NaMatrix& A, int row, int& k0, int& k1, NaScalars* sc) {
  k0 = A.row_ptr[row];
  k1 = A.row_ptr[row + 1];
  if (k0 < 0 || k1 < k0 || k1 > A.nnzb) {
    atomicMax(&sc->status, MFEM_ERR_INVALID);
    return false;
  }
  return true;
}

// The inverse of a row's diagonal block; the identity, and false, where the
// block is missing (null) or singular.
__device__ __forceinline__ bool na_inverse(const double* D, double* Di) {
  const double c00 = D ? D[4] * D[8] - D[5] * D[7] : 0.0;
  const double c01 = D ? D[5] * D[6] - D[3] * D[8] : 0.0;
  const double c02 = D ? D[3] * D[7] - D[4] * D[6] : 0.0;
  const double det = D ? D[0] * c00 + D[1] * c01 + D[2] * c02 : 0.0;
  if (det != 0.0 && std::isfinite(det)) {
    const double id = 1.0 / det;
    Di[0] = c00 * id;
    Di[1] = (D[2] * D[7] - D[1] * D[8]) * id;
    Di[2] = (D[1] * D[5] - D[2] * D[4]) * id;
    Di[3] = c01 * id;
    Di[4] = (D[0] * D[8] - D[2] * D[6]) * id;
    Di[5] = (D[2] * D[3] - D[0] * D[5]) * id;
    Di[6] = c02 * id;
    Di[7] = (D[1] * D[6] - D[0] * D[7]) * id;
    Di[8] = (D[0] * D[4] - D[1] * D[3]) * id;
    return true;
  }
#pragma unroll
  for (int e = 0; e < 9; ++e) Di[e] = (e % 4 == 0) ? 1.0 : 0.0;
  return false;
}

// D^{-1} of the diagonal blocks, r = b, z = D^{-1} b, x = 0, |b|^2, r.z.
__global__ void __launch_bounds__(kNaThreads) k_na_init(NaMatrix A, const double* b, double* x,
                                                        NaView v, int max_iters, double tol) {
  NaScalars* sc = v.sc;
  double dots[2] = {0.0, 0.0};
  const int row = blockIdx.x * kNaThreads + threadIdx.x;
  if (row < A.n) {
    int k0, k1;
    const double* D = nullptr;
    if (na_row_ok(A, row, k0, k1, sc))
      for (int k = k0; k < k1; ++k)
        if (A.col[k] == row) D = A.val + 9 * (size_t)k;
    double Di[9];
    if (!na_inverse(D, Di)) atomicMax(&sc->status, MFEM_ERR_INVALID);  // missing or singular diagonal block
#pragma unroll
    for (int e = 0; e < 9; ++e) v.dinv[9 * (size_t)row + e] = Di[e];
    double r[3] = {b[3 * row], b[3 * row + 1], b[3 * row + 2]}, z[3];
    na_prec(Di, r, z);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v.r[3 * row + c] = r[c];
      v.z[3 * row + c] = z[c];
      x[3 * row + c] = 0.0;
      dots[0] += r[c] * r[c];
      dots[1] += r[c] * z[c];
    }
  }
  na_tile_partials<2>(dots, v.partials);
  if (na_last_tile(sc)) {
    const double rr = na_sum(v.partials, 0), rz = na_sum(v.partials, 1);
    sc->rr0 = rr;
    sc->rz = rz;
    sc->beta = 0.0;
    sc->iter = 0;
    sc->max_iters = max_iters;
    sc->thr = fmax(tol * tol * rr, DBL_MIN);
    sc->err = rr == 0.0 ? 0.0 : 1.0;
    sc->active = (na_status(sc) == 0 && rr != 0.0 && rr >= sc->thr && max_iters > 0) ? 1 : 0;
    // No iteration allowed while the residual is above the threshold: the
    // solve stops on max_iters, as Eigen's NoConvergence.
    if (na_status(sc) == 0 && rr != 0.0 && rr >= sc->thr && max_iters == 0) sc->status = MFEM_ERR_CG_MAXITER;
    if (!(rr == rr) || !(rz == rz)) sc->status = MFEM_ERR_NONFINITE;
  }
}

// Ap = A p, p = z + beta p_prev (formed per column), p.Ap; alpha = rz / p.Ap.
__global__ void __launch_bounds__(kNaThreads) k_na_spmv(NaMatrix A, NaView v) {
  NaScalars* sc = v.sc;
  if (!sc->active) return;
  const int it = sc->iter;
  const double beta = sc->beta;
  const bool first = it == 0;
  const double* pin = (it & 1) ? v.p[0] : v.p[1];
  double* pout = (it & 1) ? v.p[1] : v.p[0];
  double dots[1] = {0.0};
  const int row = blockIdx.x * kNaThreads + threadIdx.x;
  if (row < A.n) {
    int k0, k1;
    double acc[3] = {0.0, 0.0, 0.0};
    if (na_row_ok(A, row, k0, k1, sc))
      for (int k = k0; k < k1; ++k) {
        const int c = A.col[k];
        if (c < 0 || c >= A.n) {
          atomicMax(&sc->status, MFEM_ERR_INVALID);
          continue;
        }
        const double* B = A.val + 9 * (size_t)k;
        double p[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) p[j] = first ? v.z[3 * c + j] : v.z[3 * c + j] + beta * pin[3 * c + j];
#pragma unroll
        for (int i = 0; i < 3; ++i) acc[i] += B[3 * i] * p[0] + B[3 * i + 1] * p[1] + B[3 * i + 2] * p[2];
      }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double p = first ? v.z[3 * row + i] : v.z[3 * row + i] + beta * pin[3 * row + i];
      pout[3 * row + i] = p;
      v.Ap[3 * row + i] = acc[i];
      dots[0] += p * acc[i];
    }
  }
  na_tile_partials<1>(dots, v.partials);
  if (na_last_tile(sc)) sc->alpha = sc->rz / na_sum(v.partials, 0);
}

// x += alpha p, r -= alpha Ap, z = D^{-1} r; then the stopping test and beta.
__global__ void __launch_bounds__(kNaThreads) k_na_update(int n, double* x, NaView v) {
  NaScalars* sc = v.sc;
  if (!sc->active) return;
  const int it = sc->iter;
  const double alpha = sc->alpha;
  const double* p = (it & 1) ? v.p[1] : v.p[0];
  double dots[2] = {0.0, 0.0};
  const int row = blockIdx.x * kNaThreads + threadIdx.x;
  if (row < n) {
    double r[3], z[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      x[3 * row + c] += alpha * p[3 * row + c];
      r[c] = v.r[3 * row + c] - alpha * v.Ap[3 * row + c];
      v.r[3 * row + c] = r[c];
      dots[0] += r[c] * r[c];
    }
    na_prec(v.dinv + 9 * (size_t)row, r, z);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v.z[3 * row + c] = z[c];
      dots[1] += r[c] * z[c];
    }
  }
  na_tile_partials<2>(dots, v.partials);
  if (na_last_tile(sc)) {
    const double rr = na_sum(v.partials, 0), rz = na_sum(v.partials, 1);
    // As in Eigen's loop, the iteration that meets the threshold is not
    // counted.
    sc->err = sqrt(rr / sc->rr0);
    if (!(rr == rr) || !(rz == rz)) {
      sc->status = MFEM_ERR_NONFINITE;
      sc->active = 0;
    } else if (na_status(sc) != 0 || rr < sc->thr) {
      sc->active = 0;
    } else {
      sc->beta = rz / sc->rz;
      sc->rz = rz;
      sc->iter = it + 1;
      if (it + 1 >= sc->max_iters) {
        sc->status = MFEM_ERR_CG_MAXITER;
        sc->active = 0;
      }
    }
  }
}

// ------------------------------------------------------ resident form ---
// One cooperative launch: a block owns up to kNaMaxSlices slices of 32 rows,
// three warps a slice (one per component, the FP64 pipe's 64 cycles an
// instruction being what the product costs), keeps their blocks in shared
// memory as planes of 32 lanes (rows by decreasing length, so that a mesh's long
// and short rows get slices of their own), and p at its rows and its halo, the
// distinct columns outside its rows, found by hashing the columns once a
// call.  The blocks exchange z and their partial sums as tagged records
// (exchange.cuh); each sums all partials itself in the same order.
//   p = z + beta p;  Ap;  (p, Ap) -> alpha;  x += alpha p;  r -= alpha Ap;
//   z = D^-1 r;  (r, r), (r, z) -> the stopping test and beta
// 9,000 rows, 109k blocks, 230 iterations: 10.9 ms with the launches (two an
// iteration, one thread summing 36 tiles' partials in turn), 2.4 ms so (10.4 us
// an iteration; 3.15 ms with the quotients and comparisons in every warp, since
// the pipe takes 19 cycles of the SM for each, and the halo's records fetched
// when they are used).  Of the 20,000 cycles the product is 5,400, the two
// exchanges of 141 blocks 6,800, trees and a division 3,000.
// A partial record is overwritten two exchanges after everybody has read it
// (two buffers by parity), z only after the exchange of (p, Ap), before which
// everybody has read it.
constexpr int kNaMaxSlices = 7;      // 32768 rows over 147 blocks
constexpr int kNaFewSlices = 3;      // up to 14592 rows over 152 blocks: no spilled registers
constexpr int kNaMaxHalo = 2560;
constexpr int kNaMaxSlots = 448;     // of a block's slices
constexpr int kNaHash = 8192;
constexpr size_t kNaSmem = 220 * 1024;
constexpr size_t kNaOffTable = 64 * (size_t)kNaMaxSlots + 4 * (size_t)kNaMaxHalo;  // li, halo columns

template <int kSlices>  // the most slices a block may have: the registers a thread may take
__global__ void __launch_bounds__(96 * kSlices) k_na_resident(NaMatrix A, const double* b, double* x, NaView v,
                                                                   int max_iters, double tol) {
  using namespace mfem_gpu;
  extern __shared__ __align__(16) unsigned char na_smem[];
  __shared__ int slot0[kNaMaxSlices + 1], nh_s, bad_s, flags;
  __shared__ int len_s[32 * kNaMaxSlices];
  __shared__ uint8_t row_at[32 * kNaMaxSlices], place_of[32 * kNaMaxSlices];
  __shared__ double part[2][kNaMaxSlices], tot[2], coef, rcp;
  const int T = blockDim.x, S = T / 96, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sl = warp / 3, comp = warp % 3, G = gridDim.x, bk = blockIdx.x;
  const int row0 = 32 * S * bk, row1 = min(A.n, row0 + 32 * S), own = 32 * S;
  const int mine = 32 * sl + lane;  // place of this thread's row in the block
  const bool lead = comp == 0;
  NaScalars* sc = v.sc;
  uint16_t* li = reinterpret_cast<uint16_t*>(na_smem);
  int* hcol = reinterpret_cast<int*>(na_smem + 64 * (size_t)kNaMaxSlots);
  unsigned seq = __ldcg(v.seq);

  // ---- the pattern: row lengths, slots of each slice
  if (threadIdx.x == 0) nh_s = bad_s = flags = 0;
  __syncthreads();
  // rows by decreasing length (the long and the short rows of a mesh in
  // slices of their own: fewer slots), rows of equal length in order
  for (int i = threadIdx.x; i < own; i += T) {
    int l = -1;
    if (row0 + i < row1) {
      const int a0 = A.row_ptr[row0 + i], a1 = A.row_ptr[row0 + i + 1];
      if (a0 < 0 || a1 < a0 || a1 > A.nnzb) bad_s = 1;
      else l = a1 - a0;
    }
    len_s[i] = l;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < own; i += T) {
    int at = 0;
    for (int j = 0; j < own; ++j) at += len_s[j] > len_s[i] || (len_s[j] == len_s[i] && j < i);
    place_of[i] = (uint8_t)at;
    row_at[at] = (uint8_t)i;
  }
  __syncthreads();
  const int row = row0 + row_at[mine];
  const bool live = row < row1 && !bad_s;
  const int len = live ? len_s[row_at[mine]] : 0, k0 = live ? A.row_ptr[row] : 0;
  int slen = len;
  for (int off = 16; off > 0; off >>= 1) slen = max(slen, __shfl_xor_sync(0xffffffffu, slen, off));
  if (lead && lane == 0) slot0[sl + 1] = slen;
  __syncthreads();
  if (threadIdx.x == 0) {
    slot0[0] = 0;
    for (int s = 0; s < S; ++s) slot0[s + 1] = min(slot0[s] + slot0[s + 1], kNaMaxSlots + 1);
    if (slot0[S] > kNaMaxSlots) bad_s = 1;
  }
  __syncthreads();
  const bool fits = !bad_s;
  const int slots = fits ? slot0[S] : 0, s_at = fits ? slot0[sl] : 0;
  const int s_len = fits ? slot0[sl + 1] - s_at : 0;
  // ---- the halo: the distinct columns outside the block's rows, hashed
  int* keys = reinterpret_cast<int*>(na_smem + kNaOffTable);
  uint16_t* at = reinterpret_cast<uint16_t*>(keys + kNaHash);
  for (int i = threadIdx.x; i < kNaHash; i += T) keys[i] = -1;
  __syncthreads();
  auto hash = [](int c) { return (int)(((unsigned)c * 2654435761u) >> 19); };  // 13 bits
  if (fits && live)
    for (int k = comp; k < len; k += 3) {
      const int c = A.col[k0 + k];
      if (c < 0 || c >= A.n) {
        bad_s = 1;
      } else if (c < row0 || c >= row1) {
        // the table holds at most kNaMaxHalo keys: a free entry is always near
        int h = hash(c);
        for (int n = 0;; ++n, h = (h + 1) & (kNaHash - 1)) {
          if (n >= 256 || *(volatile int*)&nh_s > kNaMaxHalo) {
            bad_s = 1;
            break;
          }
          const int was = atomicCAS(&keys[h], -1, c);
          if (was == -1) atomicAdd(&nh_s, 1);
          if (was == -1 || was == c) break;
        }
      }
    }
  __syncthreads();
  if (nh_s > kNaMaxHalo && threadIdx.x == 0) bad_s = 1;
  __syncthreads();
  const bool whole = !bad_s;
  __syncthreads();
  if (threadIdx.x == 0) nh_s = 0;
  __syncthreads();
  if (whole)
    for (int i = threadIdx.x; i < kNaHash; i += T)
      if (keys[i] >= 0) {
        const int j = atomicAdd(&nh_s, 1);
        at[i] = (uint16_t)j;
        hcol[j] = keys[i];
      }
  __syncthreads();
  const int nh = whole ? nh_s : 0;
  if (whole)
    for (int k = comp; k < s_len; k += 3) {
      int j = mine;  // past the row's end: the row itself, with a zero block
      if (live && k < len) {
        const int c = A.col[k0 + k];
        if (c >= row0 && c < row1) {
          j = place_of[c - row0];
        } else {
          int h = hash(c);
          while (keys[h] != c) h = (h + 1) & (kNaHash - 1);
          j = own + at[h];
        }
      }
      li[32 * (s_at + k) + lane] = (uint16_t)j;
    }
  __syncthreads();
  // ---- vectors, then as many of the slots' blocks as fit
  double* vec = reinterpret_cast<double*>(na_smem + kNaOffTable);  // p: [own + nh][3]
  double* ex = vec + 3 * (own + nh);                               // [2][S][3][32]
  double* mat = ex + 192 * S;                                      // [slot][9][32]
  const size_t left = kNaSmem - kNaOffTable - sizeof(double) * (3 * (size_t)(own + nh) + 192 * (size_t)S);
  const int res = min(slots, (int)(left / 2304));
  for (int i = warp; whole && i < res; i += T / 32) {  // a warp a slot
    int s = 0;
    while (i >= slot0[s + 1]) ++s;
    const int r = row0 + row_at[32 * s + lane], k = i - slot0[s];
    int q = -1;
    if (r < row1 && A.row_ptr[r] + k < A.row_ptr[r + 1]) q = A.row_ptr[r] + k;
#pragma unroll
    for (int e = 0; e < 9; ++e) mat[288 * (size_t)i + 32 * e + lane] = q >= 0 ? A.val[9 * (size_t)q + e] : 0.0;
  }
  // ---- D^-1 (k_na_init), r = b, z
  double D[3] = {0.0, 0.0, 0.0}, r = 0.0, z = 0.0, p = 0.0, xv = 0.0, y = 0.0;
  if (whole && live) {
    const double* Bd = nullptr;
    for (int k = 0; k < len; ++k)
      if (A.col[k0 + k] == row) Bd = A.val + 9 * (size_t)(k0 + k);
    double Di[9];
    if (!na_inverse(Bd, Di)) bad_s = 1;
#pragma unroll
    for (int c = 0; c < 3; ++c) D[c] = comp == 0 ? Di[c] : comp == 1 ? Di[3 + c] : Di[6 + c];
    const double r3[3] = {b[3 * row], b[3 * row + 1], b[3 * row + 2]};
    r = comp == 0 ? r3[0] : comp == 1 ? r3[1] : r3[2];
    z = fma(D[2], r3[2], fma(D[1], r3[1], D[0] * r3[0]));
  }

  // The sums of quantities 0 .. nq - 1, whose parts of the block's slices are
  // in part[][]: one warp per quantity sends the block's sum and adds up
  // everybody's.  `beside`: the last warp's, during the wait; `then(q, sum)`:
  // lane 0's of the warp that has the sum.  False: a wait ran out.
  auto total = [&](int nq, auto beside, auto then) -> bool {
    __syncthreads();
    if (warp < nq) {
      double t = 0.0;
      for (int s = 0; s < S; ++s) t += part[warp][s];
      if (G > 1) {
        uint4* rec = v.recs + ((seq & 1) * kMaxCopies * 2 + warp) * kNaMaxBlocks;
        const int copies = exchange_copies(G);
        if (lane < copies) st_rec(rec + lane * 2 * kNaMaxBlocks + bk, rec_of(t, seq));
        rec += (bk % copies) * 2 * kNaMaxBlocks;
        bool ok = true;
        t = fetch_sum(rec, G, seq, &sc->error, ok);
        if (!ok && lane == 0) atomicOr(&flags, 1);
      }
      if (lane == 0) {
        tot[warp] = t;
        then(warp, t);
      }
    } else if (warp == T / 32 - 1) {
      beside();
    }
    __syncthreads();
    ++seq;
    return (flags & 1) == 0;
  };
  auto slice_sum = [&](int q, double e) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) e += __shfl_down_sync(0xffffffffu, e, off);
    if (lane == 0) part[q][sl] = e;
  };
  // z to everybody; (r, r) and (r, z) in part
  auto put_rz = [&]() {
    ex[96 * sl + 32 * comp + lane] = r;
    ex[96 * S + 96 * sl + 32 * comp + lane] = z;
    if (live && G > 1) st_rec(v.pub + 3 * (size_t)row + comp, rec_of(z, seq));
    __syncthreads();
    if (comp < 2) {
      const double* q = ex + 96 * sl + lane;
      const double* o = q + (comp == 1 ? 96 * S : 0);
      slice_sum(comp, fma(q[64], o[64], fma(q[32], o[32], q[0] * o[0])));
    }
  };
  auto nothing = []() {};
  auto keep = [](int, double) {};
  auto leave = [&]() {
    if (threadIdx.x == 0) atomicAdd(v.seq, 0x100000u);  // later calls use other tags
  };

  // ---- does every block fit, is every row in order: then |b|^2 and (r, z)
  __syncthreads();
  if (lead) slice_sum(0, lane == 0 && sl == 0 && bad_s ? 1.0 : 0.0);
  if (!total(1, nothing, keep)) {
    leave();
    return;
  }
  const bool hand_back = tot[0] != 0.0;
  __syncthreads();
  put_rz();
  unsigned ztag = seq;
  if (!total(2, nothing, keep)) {
    leave();
    return;
  }
  const double rr0 = tot[0], thr = fmax(tol * tol * rr0, DBL_MIN);
  double rz = tot[1], beta = 0.0, rr_last = rr0;
  if (hand_back || !(rr0 == rr0) || !(rz == rz)) {
    if (bk == 0 && threadIdx.x == 0) *v.seq = seq;
    return;  // sc->done stays 0
  }
  bool active = rr0 != 0.0 && rr0 >= thr && max_iters > 0;
  int status = rr0 != 0.0 && rr0 >= thr && max_iters == 0 ? MFEM_ERR_CG_MAXITER : 0, it = 0;
  constexpr unsigned long long kSign = 1ull << 63, kInf = 0x7ff0000000000000ull;
  const unsigned long long thr_bits = __double_as_longlong(thr);
  // the halo's first records of this thread, under way ahead of their use
  constexpr int kAhead = kSlices > kNaFewSlices ? 1 : 4;
  int hc[kAhead];
  bool hw[kAhead];
  uint4 hv[kAhead];
#pragma unroll
  for (int j = 0; j < kAhead; ++j) {
    const int i = threadIdx.x + j * T;
    hw[j] = i < 3 * nh;
    hc[j] = hw[j] ? 3 * hcol[i / 3] + i % 3 : 0;
  }
  auto halo_ahead = [&]() {
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      if (hw[j]) hv[j] = ld_rec(v.pub + hc[j]);
  };
  halo_ahead();
  __syncthreads();
  while (active) {
    // ---- p = z + beta p: own rows, then the halo
    const bool first = it == 0;
    p = first ? z : fma(beta, p, z);
    vec[3 * mine + comp] = p;
    bool ok = poll_recs<kAhead>(hv, [&](int j) { return v.pub + hc[j]; }, hw, ztag, &sc->error);
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      if (hw[j]) {
        double* q = vec + 3 * own + threadIdx.x + j * T;
        *q = first ? rec_double(hv[j]) : fma(beta, *q, rec_double(hv[j]));
      }
    for (int i0 = 32 * warp + kAhead * T; i0 < 3 * nh; i0 += 4 * T) {  // four records a lane in flight
      bool want[4];
      uint4 w[4];
      const uint4* src[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + j * T + lane;
        want[j] = i < 3 * nh;
        src[j] = v.pub + (want[j] ? 3 * (size_t)hcol[i / 3] + i % 3 : 0);
        w[j] = ld_rec(src[j]);
      }
      ok = poll_recs<4>(w, [&](int j) { return src[j]; }, want, ztag, &sc->error) && ok;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (want[j]) {
          double* q = vec + 3 * own + i0 + j * T + lane;
          *q = first ? rec_double(w[j]) : fma(beta, *q, rec_double(w[j]));
        }
    }
    if (!__syncthreads_and(ok)) {
      leave();
      return;
    }
    // ---- Ap, (p, Ap)
    y = 0.0;
    const int here = min(s_len, max(res - s_at, 0));
    {
      const double* m = mat + 288 * (size_t)s_at + 96 * comp + lane;
      const uint16_t* l = li + 32 * s_at + lane;
#pragma unroll 4
      for (int k = 0; k < here; ++k) {
        const double* q = vec + 3 * (int)l[32 * k];
        y = fma(m[288 * k + 64], q[2], fma(m[288 * k + 32], q[1], fma(m[288 * k], q[0], y)));
      }
#pragma unroll 4
      for (int k = here; k < s_len; ++k) {
        const double* q = vec + 3 * (int)l[32 * k];
        const double* g = A.val + 9 * (size_t)(k < len ? k0 + k : k0) + 3 * comp;
        const double a0 = k < len ? g[0] : 0.0, a1 = k < len ? g[1] : 0.0, a2 = k < len ? g[2] : 0.0;
        y = fma(a2, q[2], fma(a1, q[1], fma(a0, q[0], y)));
      }
    }
    ex[96 * sl + 32 * comp + lane] = y;
    __syncthreads();
    if (lead) {
      const double* q = ex + 96 * sl + lane;
      const double* pp = vec + 3 * mine;
      slice_sum(0, fma(pp[2], q[64], fma(pp[1], q[32], pp[0] * q[0])));
    }
    if (!total(1, [&]() { if (lane == 0) rcp = 1.0 / rz; }, [&](int, double t) { coef = rz / t; })) {
      leave();
      return;
    }
    // ---- x, r, z, (r, r), (r, z)
    const double alpha = coef;
    xv = fma(alpha, p, xv);
    r = fma(-alpha, y, r);
    ex[96 * sl + 32 * comp + lane] = r;
    __syncthreads();
    {
      const double* q = ex + 96 * sl + lane;
      z = fma(D[2], q[64], fma(D[1], q[32], D[0] * q[0]));
    }
    put_rz();
    ztag = seq;
    if (!total(2, nothing, [&](int q, double t) { if (q == 1) coef = quotient_by(t, rz, rcp); })) {
      leave();
      return;
    }
    halo_ahead();
    // (comparisons take the FP64 pipe, 19 cycles a warp: as bits they don't)
    const unsigned long long rr_bits = __double_as_longlong(tot[0]), rz_bits = __double_as_longlong(tot[1]);
    rr_last = tot[0];
    // as in Eigen's loop, the iteration that meets the threshold is not counted
    if ((rr_bits & ~kSign) > kInf || (rz_bits & ~kSign) > kInf) {  // NaN
      status = MFEM_ERR_NONFINITE;
      active = false;
    } else if (rr_bits < thr_bits) {
      active = false;
    } else {
      rz = tot[1];
      ++it;
      if (it >= max_iters) {
        status = MFEM_ERR_CG_MAXITER;
        active = false;
      }
    }
    beta = coef;
  }
  if (live) x[3 * (size_t)row + comp] = xv;
  if (bk == 0 && threadIdx.x == 0) {
    sc->iter = it;
    sc->err = rr0 == 0.0 ? 0.0 : sqrt(rr_last / rr0);
    sc->status = status;
    sc->done = 1;
    *v.seq = seq;
  }
}

std::mutex g_na_mu[kNaMaxDevices];  // one per device: its scratch copy
unsigned char* g_na_base[kNaMaxDevices] = {};
int g_na_sms[kNaMaxDevices] = {};  // blocks of the resident form that fit together

bool na_device_pointer(const void* p, int dev) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) && a.device == dev;
}

}  // namespace

extern "C" int mfem_gpu_bsr_pcg_noalloc(int32_t n_block_rows, int32_t nnzb, const int32_t* row_ptr,
                                        const int32_t* col, const double* val, const double* b,
                                        double* x, int32_t max_iters, double tol, void* stream,
                                        int32_t* iterations, double* rel_residual) {
  if (iterations) *iterations = 0;
  if (rel_residual) *rel_residual = 0.0;
  if (n_block_rows < 0 || nnzb < 0 || max_iters < 0 || !(tol >= 0.0)) return MFEM_ERR_INVALID;
  if (n_block_rows > kNaMaxRows) return MFEM_ERR_CAPACITY;
  if (n_block_rows == 0) return MFEM_OK;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return MFEM_ERR_NO_DEVICE;
  }
  if (dev < 0 || dev >= kNaMaxDevices) return MFEM_ERR_CAPACITY;
  if (!na_device_pointer(row_ptr, dev) || !na_device_pointer(b, dev) || !na_device_pointer(x, dev) ||
      (nnzb > 0 && (!na_device_pointer(col, dev) || !na_device_pointer(val, dev))))
    return MFEM_ERR_INVALID;

  std::lock_guard<std::mutex> lock(g_na_mu[dev]);
  if (!g_na_base[dev]) {  // once per device: the address of the static scratch
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_na_scratch) != cudaSuccess || !p) {
      cudaGetLastError();
      return MFEM_ERR_CUDA;
    }
    // the resident form: its shared memory, and how many of its blocks fit
    int sms = 0, per_sm = 0, coop = 0;
    const unsigned int first_tag = 1;  // the records start with tag 0
    if (cudaMemcpyAsync(static_cast<unsigned char*>(p) + kNaOffSeq, &first_tag, sizeof(first_tag),
                        cudaMemcpyHostToDevice, static_cast<cudaStream_t>(stream)) != cudaSuccess ||
        cudaStreamSynchronize(static_cast<cudaStream_t>(stream)) != cudaSuccess)
      return MFEM_ERR_CUDA;
    auto ready = [&](const void* k, int slices_) {
      return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNaSmem) == cudaSuccess &&
             cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 96 * slices_, kNaSmem) == cudaSuccess &&
             per_sm > 0;
    };
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
        ready((const void*)k_na_resident<kNaFewSlices>, kNaFewSlices) &&
        ready((const void*)k_na_resident<kNaMaxSlices>, kNaMaxSlices))
      g_na_sms[dev] = per_sm > 0 ? std::min(sms, kNaMaxBlocks) : 0;
    else
      cudaGetLastError();
    g_na_base[dev] = static_cast<unsigned char*>(p);
  }
  const NaView v = na_view(g_na_base[dev]);
  const NaMatrix A{n_block_rows, nnzb, row_ptr, col, val};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int ntiles = (n_block_rows + kNaThreads - 1) / kNaThreads;
  // Launch errors are read with cudaPeekAtLastError right after this call's
  // own launches (it leaves any pending error of the caller's in place);
  // faults while the kernels run come back from cudaStreamSynchronize.
  if (cudaMemsetAsync(v.sc, 0, sizeof(NaScalars), st) != cudaSuccess) return MFEM_ERR_CUDA;
  NaScalars h{};
  // as few slices a block as leave every block an SM of its own
  const int slices = (n_block_rows + 31) / 32, sms = g_na_sms[dev];
  const int spb = sms > 0 ? (slices + sms - 1) / sms : kNaMaxSlices + 1;
  if (spb <= kNaMaxSlices) {
    void* args[] = {(void*)&A, (void*)&b, (void*)&x, (void*)&v, (void*)&max_iters, (void*)&tol};
    const cudaError_t e = cudaLaunchCooperativeKernel(spb <= kNaFewSlices ? (const void*)k_na_resident<kNaFewSlices>
                                                                          : (const void*)k_na_resident<kNaMaxSlices>,
                                                      dim3((slices + spb - 1) / spb),
                                                      dim3(96 * spb), args, kNaSmem, st);
    // refused (a stream or process that is limited to a part of the SMs): h says
    // not done, and the launches, which need no co-residency, take the system
    if (e != cudaSuccess) {
      cudaGetLastError();
    } else if (cudaMemcpyAsync(&h, v.sc, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
               cudaStreamSynchronize(st) != cudaSuccess) {
      return MFEM_ERR_CUDA;
    }
    if (h.error) return MFEM_ERR_TIMEOUT;
    if (h.done) {
      if (iterations) *iterations = h.iter;
      if (rel_residual) *rel_residual = h.err;
      return h.status;
    }
  }
  k_na_init<<<ntiles, kNaThreads, 0, st>>>(A, b, x, v, max_iters, tol);
  if (cudaPeekAtLastError() != cudaSuccess) return MFEM_ERR_CUDA;
  int launched = 0;
  for (;;) {
    if (cudaMemcpyAsync(&h, v.sc, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return MFEM_ERR_CUDA;
    if (!h.active || launched >= max_iters) break;
    const int c = max_iters - launched < kNaChunk ? max_iters - launched : kNaChunk;
    for (int k = 0; k < c; ++k) {
      k_na_spmv<<<ntiles, kNaThreads, 0, st>>>(A, v);
      k_na_update<<<ntiles, kNaThreads, 0, st>>>(n_block_rows, x, v);
    }
    if (cudaPeekAtLastError() != cudaSuccess) return MFEM_ERR_CUDA;
    launched += c;
  }
  if (iterations) *iterations = h.iter;
  if (rel_residual) *rel_residual = h.err;
  return h.status;
}
