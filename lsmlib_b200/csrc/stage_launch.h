// stage_launch.h -- type-erased arguments of the fused stage kernels.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace lsmgpu {

struct StageArgs {
  void* out;
  const void* phi_s;
  const void* phi_n;
  const void* aux[3];
  void* rhs_out;
  double* partials;
  Box gb;
  FillBox fb;
  FillBox dom;
  unsigned bc_mask;
  double inv[3];
  double dx_sq;
  const double* dt_dev;
  double dt;
  int rk_kind;
  int use_phi0;
  int fp64_policy;  // kFp64Kinks | kFp64Sign | kStochRound (FP32 form)
  unsigned sr_seed; // nonzero: stochastic rounding of the output (FP32)
  const double* defo_tab;  // kStageDeformation (see StageParams)
  int defo_off[3];
  const double* g_dev;
  // the stage input's ghost cells may be written (set by the drivers, whose
  // arrays these are): the face-shared kinds then store the boundary values
  // of bc_mask into phi_s's ghost cells and read them as stored
  int ghosts_writable;
  int tz;  // planes per block (0: stage_tz of the fill box)
};

// Tile of the stage kernels: TX x TY cells of a plane, marched over stage_tz
// planes (kStageTZ in the FP64 band form, whose flags number the tiles).
constexpr int kStageTX = 32, kStageTY = 8, kStageTZ = 16;
constexpr int kStageMaxTZ = 11;         // the longest march otherwise
constexpr int kStageMaxSplit = 4096;    // shorter marches: at most this many blocks

// a grid's z extent ends at 65535 blocks: the shortest march that covers fb
inline int least_tz(const FillBox& fb) { return (fb.n(2) - 1) / 65535 + 1; }

inline int stage_blocks(const FillBox& fb, int tz) {
  const int gx = (fb.n(0) + kStageTX - 1) / kStageTX;
  const int gy = (fb.n(1) + kStageTY - 1) / kStageTY;
  const int gz = (fb.n(2) + tz - 1) / tz;
  return gx * gy * gz;
}

// Planes a block marches: the tz of the smallest estimated time of the FP64
// pair kernels, four blocks per SM.  A block takes about tz + 2 planes (the
// window loads and the extra z faces cost two), and a plane 2.1, 2.6, 3.2 or
// 3.5 us with 1 to 4 blocks on its SM; blocks that follow one another without a
// common start take 2.75 (fitted to the reinitialization stage).  Small grids
// so get thin slabs that reach every SM, larger ones slabs that end together.
// FP32 kernels hold five or six blocks per SM (kPairBlocks) and have no fit of
// their own: the rule's choice takes up to 5 % more than the best tz from 160
// cells an axis on, 10 % at 130, and up to 43 % more (still less than 16 planes
// take, though) at 65 to 96.  Stages alone, launched back to back, in us
// (reinitialization / velocity arrays):
//                   FP64: 16 planes  best       rule     FP32: 16  best       rule
//   33^3               34 / 29    5.7 / 4.9  5.7 / 4.8    23 / 17  4.3 / 3.3  4.3 / 3.4
//   65^3               38 / 36     13 / 11    13 / 12     25 / 19  8.1 / 6.4   10 / 8.6
//   96x80x88           38 / 36     20 / 18    20 / 19     25 / 19   13 / 9.0   15 / 13
//   129x97x131         57 / 56     47 / 45    48 / 45     43 / 36   29 / 21    31 / 22
//   161x145x131        94 / 96     78 / 77    79 / 78     59 / 39   48 / 36    49 / 36
//   211x163x150       138 / 136   127 / 123  130 / 126    79 / 64   77 / 60    79 / 63
//   257^3             387 / 379   382 / 372  384 / 373   233 / 179 230 / 176  232 / 178
//   384x320x200       518 / 512   517 / 511  524 / 516   312 / 243 310 / 243  316 / 246
inline int stage_tz(const FillBox& fb) {
  constexpr int kSms = 148, kSlots = 4 * kSms;
  constexpr double kSteady = 2.75, kPlane[5] = {0.0, 2.1, 2.6, 3.2, 3.5};
  const int left = fb.n(0) % kStageTX;   // the last column's width (pair_row_bits)
  const int ly = left <= 8 ? 4 * kStageTY : left <= 16 ? 2 * kStageTY : kStageTY;
  const long tiles = (long)(fb.n(0) / kStageTX) * ((fb.n(1) + kStageTY - 1) / kStageTY) +
                     (left ? (fb.n(1) + ly - 1) / ly : 0);
  int best = kStageMaxTZ;
  if (least_tz(fb) > best) return least_tz(fb);
  double best_cost = 0.0;
  for (int tz = kStageMaxTZ; tz >= 1; tz--) {
    if (stage_blocks(fb, tz) > kStageMaxSplit) break;
    const long blocks = tiles * ((fb.n(2) + tz - 1) / tz);
    const double cost = (tz + 2) * ((double)(blocks / kSlots) * kSteady +
                                    kPlane[(blocks % kSlots + kSms - 1) / kSms]);
    if (best_cost == 0.0 || cost < best_cost) {
      best = tz;
      best_cost = cost;
    }
  }
  return best;
}
inline int stage_blocks(const FillBox& fb) { return stage_blocks(fb, stage_tz(fb)); }

// The same for the one-cell kernels (256 threads, 3 blocks per SM: 444 at a
// time), where no partials depend on it.  Thin slabs by stage_tz below 300 blocks
// of 16 planes; then the march of 6 to 16 planes whose blocks end first
// (one_cell_end); from 3 waves on 13 or 16, whichever takes fewer planes in whole
// waves, 16 where both make as many layers.  Against the best march of 18 grids of
// the middle kind (boundary values made on the fly) this rule's choice takes 2 %
// more in FP64 and 3 % in FP32, stage_tz's 5 %, 16 planes 14 % and 9 %.  In us
// (16 planes, stage_tz, this rule):
//                strict, arrays   FP64, arrays     FP32, normal speed
//   65^3           61, 37, 37      46, 28, 28       42, 27, 27
//   40x1000x40    154, 161, 144   117, 113, 104    110, 114, 105
//   200^3         404, 403, 403   279, 278, 278    240, 241, 242
constexpr int kOneCellSlots = 3 * 148;

// When the last block of a one-cell grid ends, in planes: the full layers' blocks
// in whole waves, then the rest of them beside the blocks of the (thinner) last
// layer.  A block starts in the time of half a plane in FP32 and of none in FP64;
// a plane takes 0.4 and 0.85 of its time with one and two blocks on an SM.
inline double one_cell_end(int columns, int nz, int tz, int prec) {
  constexpr double kShare[4] = {0.4, 0.4, 0.85, 1.0};
  const double start = prec == 8 ? 0.0 : 0.5;
  const int layers = (nz + tz - 1) / tz, last = nz - (layers - 1) * tz;
  const long full = (long)columns * (layers - 1);
  const long rest = full % kOneCellSlots, free = kOneCellSlots - rest;
  const long side = rest + columns < kOneCellSlots ? rest + columns : kOneCellSlots;
  const double share = kShare[(side + 147) / 148];
  const double by_full = rest ? (tz + start) * share : 0.0;
  const double by_last = (double)((columns + free - 1) / free) * (last + start) * share;
  return (double)(full / kOneCellSlots) * (tz + start) +
         (by_full > by_last ? by_full : by_last);
}

inline int one_cell_tz(const FillBox& fb, int prec = 8) {
  const int b13 = stage_blocks(fb, 13), b16 = stage_blocks(fb, 16);
  if (b16 < 300) return stage_tz(fb);
  int best = 16;
  if (b13 >= 3 * kOneCellSlots) {
    const int w13 = (b13 + kOneCellSlots - 1) / kOneCellSlots,
              w16 = (b16 + kOneCellSlots - 1) / kOneCellSlots;
    if (b13 != b16 && w16 * 18 >= w13 * 15) best = 13;
  } else {
    const int columns = stage_blocks(fb, fb.n(2)), nz = fb.n(2);
    double end = one_cell_end(columns, nz, best, prec);
    for (int tz = 15; tz >= 6; tz--) {
      const double e = one_cell_end(columns, nz, tz, prec);
      if (e < end - 1e-9) {
        best = tz;
        end = e;
      }
    }
  }
  return best > least_tz(fb) ? best : least_tz(fb);
}

// The z slabs of a host-array call (lsmgpu_normal_tvdrk3_host): slab q holds
// planes [zlo[q], zlo[q + 1]) of the fill box, cut at multiples of kStageTZ.
// Returns their number.
constexpr int kHostSlabs = 4;
inline int stage_slabs(const FillBox& fb, int zlo[kHostSlabs + 1]) {
  const int layers = (fb.n(2) + kStageTZ - 1) / kStageTZ;
  const int ns = layers < kHostSlabs ? layers : kHostSlabs;
  for (int q = 0; q < ns; q++) zlo[q] = fb.lo[2] + (int)((long)q * layers / ns) * kStageTZ;
  zlo[ns] = fb.hi[2] + 1;
  return ns;
}

// At least the blocks of any fill box inside `whole`, taken as one or cut
// along z into up to `slabs` boxes with blocks of their own.  A box of n
// planes has at most kStageMaxSplit blocks or ceil(n / kStageMaxTZ) a column
// of tiles, and each cut adds up to one layer of tiles to the sum of the latter.
inline int stage_blocks_max(const FillBox& whole, int slabs = 1) {
  FillBox w = whole;
  w.hi[2] += (slabs - 1) * (kStageMaxTZ - 1);
  return stage_blocks(w, kStageMaxTZ) + slabs * kStageMaxSplit;
}

// kind: StageKind; prec: 8 (FP64) or 4 (FP32)
cudaError_t launch_stage_strict(int kind, int prec, const StageArgs& a,
                                cudaStream_t st);
cudaError_t launch_stage_fast(int kind, int prec, const StageArgs& a,
                              cudaStream_t st);
// The boundary values of a.bc_mask into the face ghost cells of a.phi_s that
// the stencils of a.fb reach (at least 3 domain cells per axis).
cudaError_t launch_ghosts(int prec, const StageArgs& a, cudaStream_t st);
// One stage of kStageDeformation (velocity evaluated in the kernel, so both
// precisions have it) in the FP64 band form, fast arithmetic: a32 and a64 name
// the same stage over the FP32 arrays and their FP64 copies; tile_fp64[tile]
// (tiles as in stage_blocks, x fastest) = 1 computes the tile in FP64, 0 in FP32.  Both launches write
// every output cell in both precisions.  cudaErrorNotSupported when the
// two-cells-per-thread kernels do not apply (arrays of 2^31 or more cells,
// or boundary values that cannot be stored in the ghost cells).
// The FP64 launch runs on `side` (forked from st after the ghost fills by
// event ev[0], joined back by ev[1]), so that the FP64 tiles run beside the
// FP32 launch instead of after it.
cudaError_t launch_stage_band(int kind, const StageArgs& a32, const StageArgs& a64,
                              const unsigned char* tile_fp64, cudaStream_t st,
                              cudaStream_t side, cudaEvent_t ev[2]);

}  // namespace lsmgpu
