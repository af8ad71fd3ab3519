// stage_impl.cuh -- instantiation of the fused stage kernels for one
// arithmetic mode.  Included once by stage_strict.cu (STAGE_FAST = false,
// built with --fmad=false) and once by stage_fast.cu (STAGE_FAST = true, FMA).
#include <algorithm>

#include "launch.h"
#include "stage.cuh"
#include "stage_launch.h"

namespace lsmgpu {
namespace {

template <typename T>
StageParams<T> to_params(const StageArgs& a) {
  StageParams<T> p;
  p.out = (T*)a.out;
  p.phi_s = (const T*)a.phi_s;
  p.phi_n = (const T*)a.phi_n;
  p.aux0 = (const T*)a.aux[0];
  p.aux1 = (const T*)a.aux[1];
  p.aux2 = (const T*)a.aux[2];
  p.rhs_out = (T*)a.rhs_out;
  p.partials = a.partials;
  p.gb = a.gb;
  p.fb = a.fb;
  p.dom = a.dom;
  p.bc_mask = a.bc_mask;
  for (int d = 0; d < 3; d++) {
    p.inv[d] = (T)a.inv[d];
    p.fk[d] = face_const<T>(p.inv[d]);
  }
  p.dx_sq = (T)a.dx_sq;
  p.dt_dev = a.dt_dev;
  p.dt = a.dt;
  p.rk_kind = a.rk_kind;
  p.use_phi0 = a.use_phi0;
  p.fp64_policy = a.fp64_policy;
  p.sr_seed = a.sr_seed;
  p.defo_tab = a.defo_tab;
  for (int d = 0; d < 3; d++) p.defo_off[d] = a.defo_off[d];
  p.g_dev = a.g_dev;
  p.tz = a.tz ? a.tz : stage_tz(a.fb);
  return p;
}

// The boundary values of a.bc_mask can be stored in phi_s's ghost cells:
// the caller allows it, and every axis with a boundary kind has at least 3
// domain cells (so no ghost value depends on another ghost cell).
bool ghosts_storable(const StageArgs& a) {
  if (!a.ghosts_writable) return false;
  for (int d = 0; d < 3; d++) {
    const unsigned face_bits = 3u << (2 * d);
    const bool any = (a.bc_mask & (face_bits | face_bits << 8 | face_bits << 16)) != 0u;
    if (any && a.dom.n(d) < 3) return false;
  }
  return true;
}

// The boundary values of a.bc_mask into phi_s's ghost cells: the planes of
// the fill box, and the z faces its stencils reach (about 4 cells per
// thread of a z ghost plane).
template <typename T>
void launch_face_ghosts(const StageArgs& a, cudaStream_t st) {
  const int zchunks = (int)std::min<long>(
      4096, ((long)a.dom.n(0) * a.dom.n(1) + 4 * kFaceGhostThreads - 1) /
                (4 * kFaceGhostThreads));
  const long groups = (a.fb.n(2) + kGhostPlanes - 1) / kGhostPlanes;
  const long blocks = groups * face_ghost_xy_blocks(a.dom.n(0), a.dom.n(1)) + 6L * zchunks;
  launch_after(k_face_ghosts<T>, (unsigned)blocks, kFaceGhostThreads, st, (T*)a.phi_s, a.gb,
               a.dom, a.bc_mask, a.fb.lo[2], a.fb.hi[2], zchunks);
  ++launch_counter();
}

// The pair kernels take the stage: offsets fit 32 bits, and the ghost cells
// are stored (no boundary kind, or k_face_ghosts can write them first).
bool pairs_apply(const StageArgs& a) {
  const bool small = a.gb.sz() * (long)a.gb.n[2] < (1L << 31);   // 32-bit offsets
  return small && (a.bc_mask == 0u || ghosts_storable(a));
}

// One kind: a two-cells-per-thread kernel where it applies (FMA or FP32
// arithmetic; the face-shared kernel for the two-sided kinds, the one-sided
// pair kernel for the upwind kinds) and pairs_apply; else one cell per
// thread with the boundary values generated on the fly.  All cover TX x TY
// x p.tz cells per block (a narrow last column of tiles leaves blocks without
// work, which report no speed), so the grid (and the per-block CFL partials) are
// the same.
template <typename T, int KIND>
void launch_kind(dim3 grid, const StageArgs& a, const StageParams<T>& p, cudaStream_t st) {
  constexpr int TX = kStageTX, TY = kStageTY;
  static_assert(TX == kPairTX && TY == kPairTY, "one tiling for all stage kernels");
  if constexpr (UseFaces<T, KIND, STAGE_FAST, TX>::value) {
    if (pairs_apply(a)) {
      StageParams<T> q = p;
      if (a.bc_mask != 0u) {
        launch_face_ghosts<T>(a, st);
        q.bc_mask = 0u;
      }
      if constexpr (sizeof(T) == 4) {
        if (p.fp64_policy & kFp64Kinks) {
          launch_after(k_stage_pairs<T, KIND, true>, grid, kPairThreads, st, q);
          return;
        }
      }
      launch_after(k_stage_pairs<T, KIND, false>, grid, kPairThreads, st, q);
      return;
    }
  }
  if constexpr (UsePairsUp<T, KIND, STAGE_FAST, TX>::value) {
    if (pairs_apply(a)) {
      StageParams<T> q = p;
      if (a.bc_mask != 0u) {
        launch_face_ghosts<T>(a, st);
        q.bc_mask = 0u;
      }
      if constexpr (sizeof(T) == 4) {
        if (p.fp64_policy & kFp64Kinks) {
          launch_after(k_stage_pairs_up<T, KIND, true>, grid, kPairThreads, st, q);
          return;
        }
      }
      launch_after(k_stage_pairs_up<T, KIND, false>, grid, kPairThreads, st, q);
      return;
    }
  }
  // Launched as usual, so that its loads may be read-only ones (grid_wait):
  // as a dependent launch with ordinary loads the stages at 256^3 took 538 us
  // for 503 (FP64 velocity arrays, boundary values made on the fly), 708 for
  // 663 (the same in strict mode), 437 for 387 (FP32).
  StageParams<T> q = p;
  if (KIND != kStageNormalRhs && a.tz == 0) {
    q.tz = one_cell_tz(a.fb, (int)sizeof(T));
    grid.z = (a.fb.n(2) + q.tz - 1) / q.tz;
  }
  k_stage<T, KIND, STAGE_FAST, TX, TY><<<grid, dim3(TX, TY, 1), 0, st>>>(q);
}

template <typename T>
cudaError_t launch_t(int kind, const StageArgs& a, cudaStream_t st) {
  constexpr int TX = kStageTX, TY = kStageTY;
  const FillBox& fb = a.fb;
  const StageParams<T> p = to_params<T>(a);
  const dim3 grid((fb.n(0) + TX - 1) / TX, (fb.n(1) + TY - 1) / TY,
                  (fb.n(2) + p.tz - 1) / p.tz);
  switch (kind) {
    case kStageAdvect: launch_kind<T, kStageAdvect>(grid, a, p, st); break;
    case kStageNormal: launch_kind<T, kStageNormal>(grid, a, p, st); break;
    case kStageReinit: launch_kind<T, kStageReinit>(grid, a, p, st); break;
    case kStageDeformation: launch_kind<T, kStageDeformation>(grid, a, p, st); break;
    case kStageNormalRhs: launch_kind<T, kStageNormalRhs>(grid, a, p, st); break;
    default:
      return cudaErrorInvalidValue;
  }
  ++launch_counter();
  return cudaGetLastError();
}

#ifdef STAGE_BAND_FN
// the FP64 band form of one upwind kind: FP32 launch for the tiles flagged 0,
// FP64 launch for those flagged 1, each also writing the other precision
template <int KIND>
cudaError_t band_kind(dim3 grid, const StageArgs& a32, const StageArgs& a64,
                      const unsigned char* tile_fp64, cudaStream_t st, cudaStream_t side,
                      cudaEvent_t ev[2]) {
  constexpr int TX = kStageTX, TY = kStageTY;
  static_assert(UsePairsUp<float, KIND, STAGE_FAST, TX>::value &&
                    UsePairsUp<double, KIND, STAGE_FAST, TX>::value,
                "the band form runs the two-cells-per-thread upwind kernels");
  if (!pairs_apply(a32) || !pairs_apply(a64)) return cudaErrorNotSupported;
  StageParams<float> q32 = to_params<float>(a32);
  StageParams<double> q64 = to_params<double>(a64);
  if (a32.bc_mask != 0u) {
    launch_face_ghosts<float>(a32, st);
    launch_face_ghosts<double>(a64, st);
    q32.bc_mask = q64.bc_mask = 0u;
  }
  q32.tile_fp64 = q64.tile_fp64 = tile_fp64;
  q32.tile_want = 0u;
  q64.tile_want = 1u;
  q32.tz = q64.tz = kStageTZ;   // the tiles that the flags number
  q32.out_alt = a64.out;
  q64.out_alt = a32.out;
  const dim3 blk(TX / 2, TY, 1);
  cudaError_t e;
  if ((e = cudaEventRecord(ev[0], st)) != cudaSuccess ||
      (e = cudaStreamWaitEvent(side, ev[0], 0)) != cudaSuccess)
    return e;
  k_stage_pairs_up<double, KIND, false, true><<<grid, blk, 0, side>>>(q64);
  if (q32.fp64_policy & kFp64Kinks)
    k_stage_pairs_up<float, KIND, true, true><<<grid, blk, 0, st>>>(q32);
  else
    k_stage_pairs_up<float, KIND, false, true><<<grid, blk, 0, st>>>(q32);
  launch_counter() += 2;
  if ((e = cudaEventRecord(ev[1], side)) != cudaSuccess ||
      (e = cudaStreamWaitEvent(st, ev[1], 0)) != cudaSuccess)
    return e;
  return cudaGetLastError();
}
#endif

}  // namespace

#ifdef STAGE_BAND_FN
cudaError_t launch_ghosts(int prec, const StageArgs& a, cudaStream_t st) {
  if (prec == 8) launch_face_ghosts<double>(a, st);
  else launch_face_ghosts<float>(a, st);
  return cudaGetLastError();
}

cudaError_t STAGE_BAND_FN(int kind, const StageArgs& a32, const StageArgs& a64,
                          const unsigned char* tile_fp64, cudaStream_t st, cudaStream_t side,
                          cudaEvent_t ev[2]) {
  constexpr int TX = kStageTX, TY = kStageTY, TZ = kStageTZ;
  const FillBox& fb = a32.fb;
  if (fb.n(0) < 1 || fb.n(1) < 1 || fb.n(2) < 1) return cudaSuccess;
  const dim3 grid((fb.n(0) + TX - 1) / TX, (fb.n(1) + TY - 1) / TY,
                  (fb.n(2) + TZ - 1) / TZ);
  switch (kind) {
    case kStageDeformation:
      return band_kind<kStageDeformation>(grid, a32, a64, tile_fp64, st, side, ev);
    default: return cudaErrorInvalidValue;
  }
}
#endif

cudaError_t STAGE_LAUNCH_FN(int kind, int prec, const StageArgs& a,
                            cudaStream_t st) {
  if (a.fb.n(0) < 1 || a.fb.n(1) < 1 || a.fb.n(2) < 1) return cudaSuccess;
  return prec == 8 ? launch_t<double>(kind, a, st) : launch_t<float>(kind, a, st);
}

}  // namespace lsmgpu
