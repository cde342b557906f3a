// A whole PCG solve in one cooperative launch with the matrix resident in
// shared memory (k_resident.cu): the plan the host builds for a batch and the
// launch wrappers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.cuh"

namespace mfem_gpu {

// One block: a run of 32-row slices of one scene.
struct CgrBlock {
  int scene;        // slot in the batch
  int slice0, nsl;  // its slices
  int kres;         // ELL slots of each slice kept in shared memory (the rest read from L2);
                    // wide form: stages of a warp's ring
  int hoff, nh;     // its halo: columns outside its rows, CgrArgs::h_col[hoff ..]
  int loff;         // its slots' local column indices, CgrArgs::lidx[loff ..] in slot order
  int rec0, nrec;   // the scene's exchange records (tiles; slices in FP64): first, count
  int rec;          // the block's first record among them
  int row0;         // the scene's first row in the exchanged vector
  int nblk;         // blocks of the scene
  const uint8_t* pick;  // wide form: the block's slices in the warps' order, 48 (255: none)
  int spb;          // FP64: slices a block (1, 2 or 4; the last block may have fewer)
};

struct CgrArgs {
  const CgrBlock* blocks;
  const int* h_col;
  const uint16_t* lidx;
  uint4* recs;        // [parity][copy][quantity 0..2][nrec_total] tagged partial sums
  uint4* pub;         // [parity][rows (x 3 in FP64)] tagged vector
  int nrec_total;
  size_t pub_stride;  // records of one parity of pub
  unsigned int* seq;  // per scene: the next exchange's tag
  const SceneDev* sds;
  BatchCounters* ctrs;
  int max_iters;      // single-reduction form: iterations of this launch at most
};

constexpr int kCgrTile = kCgRows / 32;  // slices of a reduction tile
constexpr int kCgrMaxSlices = 16;       // slices of a block
constexpr int kCgrWideSlices = 48;      // slices of a block of the wide form
constexpr int kCgrWideWarps = 16;       // its warps, up to three slices each
constexpr unsigned kCgrStage = 1280 + 64;  // a slot in the wide form: 160 pairs and 32 local column indices
constexpr int kCgrWideTiles = 1024;     // reduction tiles of a scene in the wide form
constexpr int kCgrMaxTiles64 = 96;      // reduction tiles of an FP64 scene

// Dynamic shared memory of a block with `slots` resident slots, `own` rows
// (32 per slice) and `nh` halo columns.
constexpr size_t cgr_smem(bool fp64, bool fused, bool jacobi, size_t slots, size_t own, size_t nh) {
  const size_t w = fp64 ? 8 : 4;
  size_t b = slots * (288 * w + 64);                  // 9 planes and the column indices
  b += fp64 ? 24 * (own + nh) : 16 * (own + nh);      // the multiplied vector
  if (fp64) b += 120 * own;                           // exchange between the warps of a slice
  if (fused) b += 16 * nh + (jacobi ? 0 : 16 * nh + 36 * nh);
  return b;
}
// .. of the wide form: u at the rows and the halo, the halo's columns, and every
// warp's ring of `stages` slots with a barrier each.
constexpr size_t cgr_wide_smem(size_t stages, size_t own, size_t nh) {
  return 16 * (own + nh) + 16 * ((nh + 3) / 4) + kCgrWideWarps * stages * (kCgrStage + 8);
}
constexpr size_t kCgrSmem = 218 * 1024;  // dynamic shared memory a block may take
constexpr int cgr_threads(bool fp64, int spb) { return fp64 ? 384 : (spb > 8 ? 512 : 256); }
constexpr int kCgrMaxSpb64 = 4;  // twelve warps: 3 components x 4, 2 or 1 parts of the slots

// Blocks per SM that can be resident with this much dynamic shared memory.
int cgr_blocks_per_sm(bool fp64, bool fused, bool jacobi, bool wide, int threads, size_t smem);
// The solve of every active scene.  fused: the single-reduction iteration
// (mixed path), up to args.max_iters iterations or until a scene's stop is to
// be verified; else Eigen's two-reduction iteration to its end.
cudaError_t launch_cgr(const CgrArgs& args, bool fp64, bool fused, bool jacobi, bool wide, int nblocks, int threads,
                       size_t smem, cudaStream_t stream);

}  // namespace mfem_gpu
