// distance.cu -- signed distance function on the GPU with the values of the
// reference's fast marching method (computeDistanceFunction3d,
// src/serial/lsm_FMM_field_extension.c, src/toolbox/fast_marching_method).
//
// The reference marches a heap.  The front (points on or next to the zero
// level set) is initialised and marked KNOWN first; then the trial point of
// smallest |d| is accepted, one at a time, and every acceptance recomputes
// the trial values of its neighbours from all KNOWN points around them
// (:1021-1119 first order, :1232-1381 second order).  A point's final value
// is therefore the update over
//   - all its front neighbours,
//   - the free neighbours accepted before it,
//   - at second order, the next point along an axis when it is a front
//     point or was accepted before the neighbour whose acceptance made the
//     last update.
// "Accepted before" is decided by acceptance time (Time3 below): mostly the
// heap accepts in order of |d|, but an acceptance can lower a trial
// neighbour's value below the key just popped (the second-order update is
// not monotone), and the heap then pops that neighbour next.
// The GPU computes the march's result as the fixed point of these rules,
// without a heap:
//   1. the front is initialised cell by cell exactly as the reference does
//      (:397-668);
//   2. every other point starts unreached; passes over a band of active
//      points (below) evaluate the rules until nothing changes;
//   3. points no front reaches keep the reference's default -1; points with
//      mask < 0 are outside the domain and hold LSMLIB_REAL_MAX.
// Built with --fmad=false so the update rounds as the reference's C does.
// "Before" is the order of (acceptance time, linear point index): the time
// decides, and the index breaks exact ties.  Where no two keys tie this is
// the heap's pop order.  Where keys tie exactly (symmetric inputs, flat
// fronts, quantised data) the reference's binary heap pops the tied points in
// an order set by its whole history of insertions and removals, which no
// rule over a neighbourhood can reproduce; there the result is that of the
// same march popping ties by index.
#include <cfloat>
#include <climits>
#include <cmath>
#include <string>

#include "capi_common.h"
#include "launch.h"

using namespace lsmgpu;

namespace {

enum : unsigned char { kOutside = 0, kFront = 1, kFree = 2 };
constexpr double kZeroTol = 1.0e-11;   // LSMLIB_ZERO_TOL of the FP64 build

// Acceptance time of a free point, compared lexicographically.  A point the
// heap pops with the largest key so far (a "root") has time (|d|, -1, -1).
// A point an acceptance lowered below the keys already popped is popped
// right after its trigger (the last neighbour accepted before it), ahead of
// every larger key: its time extends the trigger's by its own |d| at the
// first level where |d| exceeds the trigger's key -- (a, |d|, -1) under a
// root trigger, (a, b, |d|) when it drops below a lowered trigger's key b.
// A time therefore always follows its trigger's.  Deeper lowering (below a
// third-level key) keeps the trigger's time; it has not been seen in
// practice.
struct Time3 {
  double a, b, c;
};

__device__ __forceinline__ bool tless(const Time3& x, const Time3& y) {
  return x.a < y.a || (x.a == y.a && (x.b < y.b || (x.b == y.b && x.c < y.c)));
}

// point x (time tx, linear index ix) is accepted before point y: by time,
// exact ties by index
__device__ __forceinline__ bool kless(const Time3& tx, long ix, const Time3& ty, long iy) {
  if (tless(tx, ty)) return true;
  if (tless(ty, tx)) return false;
  return ix < iy;
}
// the same out of line, for the rare comparisons of times whose first levels tie
__device__ __noinline__ bool kless_tied(Time3 tx, long ix, Time3 ty, long iy) {
  return kless(tx, ix, ty, iy);
}

// What an evaluation reads of a point: its value and the first level of its
// time, with kKeyFront for a front point and kKeyOutside outside the domain
// (times are >= 0) -- one 16-byte load in place of the value, the time and
// the status byte.  The time's other levels lie in an array of their own.
constexpr double kKeyFront = -1.0, kKeyOutside = -2.0;
__device__ __forceinline__ bool key_inside(double k) { return k > -1.5; }

// The whole time of a free point.  (Values that other SMs write during the
// march are loaded from L2, since an L1 line may predate the write.)
__device__ __forceinline__ Time3 time_of(const double2* vk, const double2* tm, long o) {
  const double2 bc = __ldcg(tm + o);
  return Time3{__ldcg(vk + o).y, bc.x, bc.y};
}

// linear index of the k-th point (k = 1, 2) from o in slot q's direction
__device__ __forceinline__ long nb_index(long o, const long s[3], int q, int k) {
  return o + ((q & 1) ? k : -k) * s[q >> 1];
}

// the time of a point with key ``a`` whose trigger has time ``x`` (no free
// trigger: a root)
__device__ __forceinline__ Time3 tafter(const Time3& x, double a, bool has_trigger) {
  if (!has_trigger || a > x.a) return Time3{a, -1.0, -1.0};
  if (x.b < 0 || a > x.b) return Time3{x.a, a, -1.0};
  if (x.c < 0 || a > x.c) return Time3{x.a, x.b, a};
  return x;
}

// Extension fields carried by one solve (computeExtensionFields3d): output
// fields, their source fields, the optional extension mask.
constexpr int kMaxFields = 8;
struct ExtSet {
  double* ext[kMaxFields];
  const double* src[kMaxFields];
  const double* emask;
  int nf;
};

// FMM_initializeFront_FieldExtension3d_Order1 (lsm_FMM_field_extension.c:
// 397-668) for one point; the neighbours' phi is read whatever their mask.
// Extension fields: every value starts at -1 (LSMLIB_REAL_MAX outside the
// mask); on the interface the source value; next to it the average over
// the axes of the source interpolated linearly to the nearer crossing (or
// taken from one side where the extension mask is < 0), weights
// 1/d_axis^2 (:524-660).
__global__ void k_fmm_front(double* d, double2* tm, unsigned char* st, const double* phi,
                            const double* mask, int nx, int ny, int nz, double dx,
                            double dy, double dz, ExtSet X) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  const int n[3] = {nx, ny, nz};
  const double h[3] = {dx, dy, dz};
  for (int k = blockIdx.z; k < nz; k += gridDim.z) {
    const long o = (long)i + (long)nx * ((long)j + (long)ny * k);
    tm[o] = make_double2(INFINITY, INFINITY);
    if (mask && mask[o] < 0) {
      st[o] = kOutside;
      d[o] = DBL_MAX;
      for (int k = 0; k < X.nf; k++) X.ext[k][o] = DBL_MAX;
      continue;
    }
    const double pc = phi[o];
    if (fabs(pc) < kZeroTol) {           // on the interface
      st[o] = kFront;
      d[o] = pc > 0 ? kZeroTol : -kZeroTol;
      for (int k = 0; k < X.nf; k++) X.ext[k][o] = X.src[k][o];
      continue;
    }
    const int c[3] = {i, j, k};
    const long s[3] = {1L, (long)nx, (long)nx * ny};
    bool borders = false;
    double sum = 0;
    double fsum[kMaxFields];
#pragma unroll
    for (int f = 0; f < kMaxFields; f++) fsum[f] = 0;
    for (int dir = 0; dir < 3; dir++) {
      double dist_plus = DBL_MAX, dist_minus = DBL_MAX;
      double frac_plus = 0, frac_minus = 0;
      if (c[dir] - 1 >= 0) {
        const double pm = phi[o - s[dir]];
        if (pm * pc <= 0) {
          dist_minus = pc / (pc - pm);
          frac_minus = dist_minus;
          dist_minus *= h[dir];
        }
      }
      if (c[dir] + 1 < n[dir]) {
        const double pp = phi[o + s[dir]];
        if (pp * pc <= 0) {
          dist_plus = pc / (pc - pp);
          frac_plus = dist_plus;
          dist_plus *= h[dir];
        }
      }
      if (dist_plus < DBL_MAX || dist_minus < DBL_MAX) {
        borders = true;
        const bool use_plus = dist_plus < dist_minus;
        const double dd = use_plus ? dist_plus : dist_minus;
        const double w = 1 / dd / dd;
        sum += w;
        const long on = use_plus ? o + s[dir] : o - s[dir];
        const double frac = use_plus ? frac_plus : frac_minus;
#pragma unroll
        for (int f = 0; f < kMaxFields; f++) {
          if (f >= X.nf) break;
          const double cur = X.src[f][o];
          double v;
          if (X.emask && X.emask[o] < 0) v = X.src[f][on];
          else if (X.emask && X.emask[on] < 0) v = cur;
          else v = cur + frac * (X.src[f][on] - cur);
          fsum[f] += v * w;
        }
      }
    }
    if (borders) {
      st[o] = kFront;
      d[o] = pc > 0 ? sqrt(1.0 / sum) : -sqrt(1.0 / sum);
#pragma unroll
      for (int f = 0; f < kMaxFields; f++)
        if (f < X.nf) X.ext[f][o] = fsum[f] / sum;
    } else {
      st[o] = kFree;
      d[o] = pc > 0 ? INFINITY : -INFINITY;
      for (int f = 0; f < X.nf; f++) X.ext[f][o] = -1.0;
    }
  }
}

// The Eikonal solver's data (solveEikonalEquation3d): the speed F and the
// input phi, whose values the points never updated keep.  speed == nullptr
// for the distance function.
struct Eik {
  const double* speed;
  const double* phi0;
};

// FMM_initializeFront_Eikonal3d (lsm_FMM_eikonal.c:259-312) and the domain
// marking before it (:214-246): points with mask < 0 or speed < 1e-11 are
// outside the domain and get LSMLIB_REAL_MAX; points with phi > -1e-11 are
// the front, KNOWN with their own values; the others start unreached.
__global__ void k_eik_front(double* d, double2* tm, unsigned char* st, const double* phi0,
                            const double* speed, const double* mask, long n) {
  for (long o = blockIdx.x * (long)blockDim.x + threadIdx.x; o < n;
       o += (long)gridDim.x * blockDim.x) {
    tm[o] = make_double2(INFINITY, INFINITY);
    if ((mask && mask[o] < 0) || speed[o] < kZeroTol) {
      st[o] = kOutside;
      d[o] = DBL_MAX;
    } else if (phi0[o] > -kZeroTol) {
      st[o] = kFront;
      d[o] = phi0[o];
    } else {
      st[o] = kFree;
      d[o] = INFINITY;
    }
  }
}

// A point's update: its value and acceptance time, and per axis what it took
// (the side, -1: none; the value there; the next point's value where the
// second-order stencil holds).
struct Update {
  double val;
  Time3 t;
  int side[3];
  bool second[3];
  double u1[3], u2[3];
};

// The neighbours of one point, by slot 2*axis + (plus side): the immediate
// neighbour (value v1, time t1) and, at second order, the next one in that
// direction (v2, t2).
struct Stencil {
  double v1[6], v2[6];
  Time3 t1[6], t2[6];
  unsigned char has1, front1, has2, front2;  // bit per slot
};

// The coefficients of the reference's trial update (:1021-1119 first order,
// :1232-1381 second order) over the immediate neighbours in ``incl`` (bit
// per slot), accumulated in its order and rounding.  Per axis the minus
// neighbour is taken when included and replaced by the plus one when its
// |d| is strictly smaller.  At second order the next point in the chosen
// direction counts when it was KNOWN at the update -- a front point, or a
// free point accepted before the trigger (time ``trig``, index ``itrig``;
// the front phase comes before every free point) -- and its |d| is not above
// the neighbour's.  ``cterm`` is what the constant term loses: 1 for the
// distance function, 1/F^2 for the Eikonal solver (lsm_FMM_eikonal.c:427,
// :621).  Returns the discriminant B^2 - 4AC.
template <int ORDER>
__device__ __forceinline__ double fmm_coeffs(const Stencil& n, int incl,
                                             const Time3& trig, long itrig, bool has_trigger,
                                             long o, const long s3[3], const double i2[3],
                                             double cterm, double& A, double& B) {
  double C = 0;
  A = 0;
  B = 0;
#pragma unroll
  for (int dir = 0; dir < 3; dir++) {
    double u1 = DBL_MAX, u2 = DBL_MAX;
    int sw = 0;
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const int q = 2 * dir + side;
      if (!(incl & (1 << q))) continue;
      if (side == 1 && !(fabs(n.v1[q]) < fabs(u1))) continue;
      u1 = n.v1[q];
      u2 = DBL_MAX;
      sw = 0;
      if (ORDER == 2 && (n.has2 & (1 << q)) && fabs(n.v2[q]) <= fabs(u1) &&
          ((n.front2 & (1 << q)) ||
           (has_trigger && kless(n.t2[q], nb_index(o, s3, q, 2), trig, itrig)))) {
        u2 = n.v2[q];
        sw = 1;
      }
    }
    if (!(u1 < DBL_MAX)) continue;
    const double inv = i2[dir];
    if (ORDER == 1) {
      A += inv;
      B += inv * u1;
      C += inv * u1 * u1;
    } else {
      const double s = 1.0 + 0.5 * sw;
      const double contrib = sw == 1 ? 2.0 * u1 - 0.5 * u2 : u1;
      A += inv * s * s;
      B += inv * s * contrib;
      C += inv * contrib * contrib;
    }
  }
  B *= -2.0;
  C -= cterm;
  return B * B - 4.0 * A * C;
}

// The root the reference takes (disc >= 0), in its rounding: by the sign
// of B for the distance function (lsm_FMM_field_extension.c:1106-1117), the
// larger root for the Eikonal solver (lsm_FMM_eikonal.c:433-436).
template <bool EIK>
__device__ __forceinline__ double fmm_root(double A, double B, double disc) {
  if (EIK) return 0.5 * (-B + sqrt(disc)) / A;
  if (B == 0) return 0;
  if (B < kZeroTol) return 0.5 * (-B + sqrt(disc)) / A;
  return 0.5 * (-B - sqrt(disc)) / A;
}

// ---- the band solver ----------------------------------------------------------
// The threshold T on acceptance time (its first level) advances in steps; a
// point's value is stored only while its time is within T.  A point depends
// only on points with earlier times, so the points within T settle exactly
// and are never revised once T has moved past them: the work follows a thin
// band, as the march does, instead of relaxing the whole grid.  Each pass
// evaluates the points of the active list, one thread per point, from its
// neighbours' current values; a point whose value or time changed queues
// the points whose stencil reads it for the next pass.  A point whose time
// is above T keeps its time as a candidate and waits in a pending list;
// when a pass queues nothing, T moves to max(T + delta, smallest
// candidate) and the pending points it reaches are queued.  All passes run
// in one kernel, k_fmm_march, whose blocks meet twice a pass: every queued
// point is evaluated from the values before the pass and its readers queued;
// then the changes are stored.

// The threshold advances by this many of the smallest spacing per step.  A
// longer step takes fewer passes and revises its points more often: 6 cells
// where the lists leave threads idle and a pass costs its latency (measured
// before a point's value and key became one load: 301x237,
// order 1: 571 passes of 10.5 us with 2 cells, 405 of 11.3 with 6; 64^3: 256
// and 228 of 14.0), 2 where they fill the GPU (128x112x120, order 2: 16.8 ms
// against 20.6 with 6).
constexpr double kDeltaCells = 2.0, kDeltaCellsSmall = 6.0;

// The value and acceptance time of free point o from its neighbours' current
// values and times: the reference's last trial update.  Every front point is
// KNOWN before the march starts (FMM_Core.c:203-243), so the front
// neighbours are always in the update.  The free neighbours are taken in
// order of time; each is in the update when the heap accepted it while this
// point was still a trial point, i.e. before this point's time as given by
// the neighbours taken so far.  The set must also be consistent with the
// point's final time -- every neighbour in it accepted before the point --
// as it always is in a real march; when it is not (a transient state of the
// passes), the set is cut before the earliest offending neighbour and the
// update is taken again.  A negative discriminant keeps the previous value:
// -1 (the reference's default) when there is none, or for the Eikonal
// solver the point's input.  Neighbours off the grid
// are left out, as the reference's bounds checks do.
template <int ORDER, bool EIK>
__device__ __noinline__ bool fmm_point(const double2* vk, const double2* tm, long o, int c0,
                                       int c1, int c2, int nx, int ny, int nz, double i2x,
                                       double i2y, double i2z, Eik E, Update* U) {
  const int c[3] = {c0, c1, c2}, n[3] = {nx, ny, nz};
  const long s[3] = {1L, (long)nx, (long)nx * ny};
  const double i2[3] = {i2x, i2y, i2z};
  Stencil nb;
  // every load first, at in-range addresses (the point itself stands in
  // for a neighbour off the grid), so that they are in flight together
  double s1[6], s2[6];
  bool in1[6], in2[6];
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const int dir = q >> 1;
    const int sg = (q & 1) ? 1 : -1;
    in1[q] = c[dir] + sg >= 0 && c[dir] + sg < n[dir];
    const long o1 = in1[q] ? o + sg * s[dir] : o;
    const double2 p1 = __ldcg(vk + o1);
    s1[q] = p1.y;
    nb.v1[q] = p1.x;
    const double2 bc1 = __ldcg(tm + o1);
    nb.t1[q] = Time3{p1.y, bc1.x, bc1.y};
    if (ORDER == 2) {
      in2[q] = in1[q] && c[dir] + 2 * sg >= 0 && c[dir] + 2 * sg < n[dir];
      const long o2 = in2[q] ? o + 2 * sg * s[dir] : o;
      const double2 p2 = __ldcg(vk + o2);
      s2[q] = p2.y;
      nb.v2[q] = p2.x;
      const double2 bc2 = __ldcg(tm + o2);
      nb.t2[q] = Time3{p2.y, bc2.x, bc2.y};
    }
  }
  nb.has1 = nb.front1 = nb.has2 = nb.front2 = 0;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const bool k1 = in1[q] && key_inside(s1[q]) && fabs(nb.v1[q]) <= DBL_MAX;
    if (!k1) {
      nb.v1[q] = DBL_MAX;
      nb.t1[q] = Time3{INFINITY, INFINITY, INFINITY};
      continue;
    }
    nb.has1 |= 1 << q;
    if (s1[q] < 0) {
      nb.front1 |= 1 << q;
      nb.t1[q] = Time3{INFINITY, INFINITY, INFINITY};
    }
    if (ORDER == 2) {
      const bool k2 = in2[q] && key_inside(s2[q]) && fabs(nb.v2[q]) <= DBL_MAX;
      if (!k2) {
        nb.v2[q] = DBL_MAX;
        continue;
      }
      nb.has2 |= 1 << q;
      if (s2[q] < 0) nb.front2 |= 1 << q;
    }
  }
  if (!nb.has1) return false;
  const int free1 = nb.has1 & ~nb.front1;
  const double cterm = EIK ? 1 / E.speed[o] / E.speed[o] : 1.0;
  const double none = EIK ? E.phi0[o] : -1.0;   // the value without an update
  // only neighbours before this (time, index)
  Time3 cap{INFINITY, INFINITY, INFINITY};
  long icap = LONG_MAX;
  for (;;) {
    int incl = nb.front1;
    bool have = incl != 0, trig_free = false;
    Time3 trig{-INFINITY, -1.0, -1.0};
    long itrig = -1;
    double cur = none;
    if (have) {
      double A, B;
      const double disc =
          fmm_coeffs<ORDER>(nb, incl, trig, itrig, false, o, s, i2, cterm, A, B);
      if (disc >= 0) cur = fmm_root<EIK>(A, B, disc);
    }
    for (int rem = free1; rem;) {
      // the earliest remaining free neighbour
      int best = -1;
      Time3 bt{INFINITY, INFINITY, INFINITY};
      long ib = LONG_MAX;
#pragma unroll
      for (int q = 5; q >= 0; q--) {
        if (!(rem & (1 << q))) continue;
        const long iq = nb_index(o, s, q, 1);
        if (best < 0 || kless(nb.t1[q], iq, bt, ib)) {
          best = q;
          bt = nb.t1[q];
          ib = iq;
        }
      }
      rem &= ~(1 << best);
      if (!kless(bt, ib, cap, icap)) break;
      if (have && !kless(bt, ib, tafter(trig, fabs(cur), trig_free), o)) break;
      incl |= 1 << best;
      trig = bt;
      itrig = ib;
      trig_free = true;
      double A, B;
      const double disc =
          fmm_coeffs<ORDER>(nb, incl, trig, itrig, true, o, s, i2, cterm, A, B);
      if (disc >= 0) cur = fmm_root<EIK>(A, B, disc);
      have = true;
    }
    const Time3 t = tafter(trig, fabs(cur), trig_free);
    // the earliest neighbour in the set not accepted before the point
    bool bad = false;
    Time3 badt{INFINITY, INFINITY, INFINITY};
    long ibad = LONG_MAX;
#pragma unroll
    for (int q = 0; q < 6; q++) {
      if (!(incl & free1 & (1 << q))) continue;
      const long iq = nb_index(o, s, q, 1);
      if (!kless(nb.t1[q], iq, t, o) && kless(nb.t1[q], iq, badt, ibad)) {
        bad = true;
        badt = nb.t1[q];
        ibad = iq;
      }
    }
    if (!bad) {
      U->val = cur;
      U->t = t;
#pragma unroll
      for (int dir = 0; dir < 3; dir++) {
        U->side[dir] = -1;
        U->second[dir] = false;
        U->u1[dir] = U->u2[dir] = DBL_MAX;
#pragma unroll
        for (int side = 0; side < 2; side++) {
          const int q = 2 * dir + side;
          if (!(incl & (1 << q))) continue;
          if (side == 1 && !(fabs(nb.v1[q]) < fabs(U->u1[dir]))) continue;
          U->side[dir] = side;
          U->u1[dir] = nb.v1[q];
          U->second[dir] = ORDER == 2 && (nb.has2 & (1 << q)) && fabs(nb.v2[q]) <= fabs(nb.v1[q]) &&
                           ((nb.front2 & (1 << q)) ||
                            (trig_free && kless(nb.t2[q], nb_index(o, s, q, 2), trig, itrig)));
          U->u2[dir] = U->second[dir] ? nb.v2[q] : DBL_MAX;
        }
      }
      return true;
    }
    cap = badt;
    icap = ibad;
  }
}

// fmm_point for nearly every point, without most of its work.  Of 26 M
// evaluations (128x112x120, order 2) none was taken twice, 0.002 % met a
// negative discriminant and 0.03 % a lowered time, but each took 2.6 roots (a
// square root and a division) to decide which neighbours come before the
// value, and some 3000 instructions in a row.  Here
//   - of a neighbour only its value and the first level of its time are read,
//     as one pair; the other levels when two tie;
//   - "a neighbour of key x comes before |value|" is read off the sign of the
//     quadratic at x where it is clear of rounding, and the root is taken once
//     at the end;
//   - whatever is unusual (a lowered or tied time of the point itself, a
//     negative or undefined discriminant, a vanishing linear term, for the
//     Eikonal solver a negative value) is left to fmm_point.
// Returns 1 with the update, 0 for a point no neighbour reaches, -1 for a
// point left to fmm_point; ``readers``: the free points whose stencil reads
// this one (bit ORDER * slot, and at second order the next for the point
// behind).  The arithmetic of the coefficients and of the root is fmm_coeffs'
// and fmm_root's.
template <int ORDER, bool EIK>
__device__ __forceinline__ int fmm_point_fast(const double2* vk, const double2* tm, long o,
                                              const int c[3], const int n[3], const long s[3],
                                              const double i2[3], const Eik& E, Update& U,
                                              unsigned& readers) {
  double v1[6], k1[6], v2[6], k2[6];
  unsigned in1 = 0, in2 = 0;
  const double cterm = EIK ? 1 / E.speed[o] / E.speed[o] : 1.0;
  // every load first, at in-range addresses, as in fmm_point
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const int dir = q >> 1, sg = (q & 1) ? 1 : -1;
    const int a1 = c[dir] + sg, a2 = c[dir] + 2 * sg;
    const bool i1 = a1 >= 0 && a1 < n[dir];
    const long o1 = i1 ? o + sg * s[dir] : o;
    in1 |= (unsigned)i1 << q;
    const double2 p1 = __ldcg(vk + o1);
    v1[q] = p1.x;
    k1[q] = p1.y;
    if (ORDER == 2) {
      const bool b2 = a2 >= 0 && a2 < n[dir];
      const long o2 = b2 ? o + 2 * sg * s[dir] : o;
      in2 |= (unsigned)b2 << q;
      const double2 p2 = __ldcg(vk + o2);
      v2[q] = p2.x;
      k2[q] = p2.y;
    }
  }
  // masks, a bit per slot: in the update so far (the fronts), waiting (the
  // free neighbours, their keys in k1), the second point usable at once
  // (a front) or once accepted before the trigger; a bit per axis: the plus
  // side is the smaller
  unsigned incl = 0, rem = 0, sec = 0, dyn = 0, plus_less = 0;
  readers = 0;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const bool has = (in1 >> q & 1) && key_inside(k1[q]) && fabs(v1[q]) <= DBL_MAX;
    const bool front = has && k1[q] < 0;
    readers |= (unsigned)((in1 >> q & 1) && !(k1[q] < 0)) << (q * ORDER);
    incl |= (unsigned)front << q;
    rem |= (unsigned)(has && !front) << q;
    if (!(has && !front)) k1[q] = INFINITY;
    if (ORDER == 2) {
      const bool has2 = has && (in2 >> q & 1) && key_inside(k2[q]) &&
                        fabs(v2[q]) <= fabs(v1[q]);
      const bool front2 = has2 && k2[q] < 0;
      readers |= (unsigned)((in2 >> q & 1) && !(k2[q] < 0)) << (2 * q + 1);
      sec |= (unsigned)front2 << q;
      dyn |= (unsigned)(has2 && !front2) << q;
    }
  }
#pragma unroll
  for (int dir = 0; dir < 3; dir++)
    plus_less |= (unsigned)(fabs(v1[2 * dir + 1]) < fabs(v1[2 * dir])) << dir;
  if (!(incl | rem)) return 0;
  double trig = -INFINITY;   // key of the last free neighbour taken
  int qtrig = -1;
  double A = 0, B = 0, C = 0, disc = 0;
  unsigned used = 0, plus = 0, second = 0;   // a bit per axis, of the update so far
  for (;;) {
    if (incl) {
      unsigned now = sec;
      if (ORDER == 2) {
        unsigned tie = 0;
#pragma unroll
        for (int q = 0; q < 6; q++) {
          now |= (dyn >> q & 1 & (unsigned)(k2[q] < trig)) << q;
          tie |= (dyn >> q & 1 & (unsigned)(k2[q] == trig)) << q;
        }
        if (tie) {
          const long it = nb_index(o, s, qtrig, 1);
#pragma unroll
          for (int q = 0; q < 6; q++)
            if (tie >> q & 1) {
              const long iq = nb_index(o, s, q, 2);
              if (kless_tied(time_of(vk, tm, iq), iq, time_of(vk, tm, it), it)) now |= 1u << q;
            }
        }
      }
      used = plus = second = 0;
      A = B = C = 0;
#pragma unroll
      for (int dir = 0; dir < 3; dir++) {
        const unsigned m = incl >> (2 * dir) & 3;
        const bool pl = m == 2 || (m == 3 && (plus_less >> dir & 1));
        const double u1 = pl ? v1[2 * dir + 1] : v1[2 * dir];
        const double inv = i2[dir];
        double a, b, g;
        if (ORDER == 1) {
          a = inv;
          b = inv * u1;
          g = inv * u1 * u1;
        } else {
          const bool sw = now >> (2 * dir + pl) & 1;
          const double u2 = pl ? v2[2 * dir + 1] : v2[2 * dir];
          const double w = sw ? 1.5 : 1.0;
          const double contrib = sw ? 2.0 * u1 - 0.5 * u2 : u1;
          a = inv * w * w;
          b = inv * w * contrib;
          g = inv * contrib * contrib;
          second |= (unsigned)sw << dir;
        }
        used |= (unsigned)(m != 0) << dir;
        plus |= (unsigned)pl << dir;
        // (x + 0 = x for the sums' values; an axis that is not used may hold anything)
        A += m ? a : 0.0;
        B += m ? b : 0.0;
        C += m ? g : 0.0;
      }
      B *= -2.0;
      C -= cterm;
      disc = B * B - 4.0 * A * C;
      if (!(disc >= 0) || !(fabs(B) > 1e-9) || (EIK && B > 0)) return -1;
    }
    if (!rem) break;
    // the earliest remaining free neighbour
    double x;
    {
      const double a = k1[0] < k1[1] ? k1[0] : k1[1], b = k1[2] < k1[3] ? k1[2] : k1[3],
                   e = k1[4] < k1[5] ? k1[4] : k1[5];
      x = a < b ? a : b;
      x = x < e ? x : e;
    }
    unsigned eq = 0;
#pragma unroll
    for (int q = 0; q < 6; q++) eq |= (unsigned)(k1[q] == x) << q;
    eq &= rem;
    if (!eq) return -1;   // an undefined key
    if (incl) {
      // x against |value|, the outer root of A u^2 - |B| u + C
      const double ax = A * x, bx = fabs(B);
      const double f = (ax - bx) * x + C;
      const double clear = 1e-12 * ((ax + bx) * x + fabs(C));
      if (!(f < -clear)) {
        if (f > clear && 2.0 * ax > bx) break;
        const double r = fabs(fmm_root<EIK>(A, B, disc));
        if (x > r) break;
        if (!(x < r)) return -1;
      }
    }
    if (eq & (eq - 1)) {   // equal keys: the whole times decide, then the indices
      int best = -1;
      for (unsigned m = eq; m; m &= m - 1) {
        const int q = __ffs(m) - 1;
        const long iq = nb_index(o, s, q, 1), ib = nb_index(o, s, best < 0 ? q : best, 1);
        if (best < 0 || kless_tied(time_of(vk, tm, iq), iq, time_of(vk, tm, ib), ib)) best = q;
      }
      eq = 1u << best;
    }
#pragma unroll
    for (int q = 0; q < 6; q++)
      if (eq >> q & 1) k1[q] = INFINITY;
    rem &= ~eq;
    incl |= eq;
    trig = x;
    qtrig = __ffs(eq) - 1;
  }
  U.val = fmm_root<EIK>(A, B, disc);
  const double t = fabs(U.val);
  if (!(t > trig)) return -1;
  U.t = Time3{t, -1.0, -1.0};
#pragma unroll
  for (int dir = 0; dir < 3; dir++) {
    const bool pl = plus >> dir & 1;
    U.side[dir] = (used >> dir & 1) ? pl : -1;
    U.second[dir] = ORDER == 2 && (second >> dir & 1);
    U.u1[dir] = pl ? v1[2 * dir + 1] : v1[2 * dir];
    U.u2[dir] = ORDER == 2 ? (pl ? v2[2 * dir + 1] : v2[2 * dir]) : DBL_MAX;
  }
  return 1;
}

// The extension fields of the point's last trial update: over the axes in
// the update, the weighted average of the upwind neighbour's field with
// weights (dist - phi_upwind)/dx^2, or (1.5 dist - 2 phi_upwind1 +
// 0.5 phi_upwind2)/dx^2 where the second-order stencil is used
// (lsm_FMM_field_extension.c:1135-1168, :1400-1460); its value is the
// update's distance (the previous one where the discriminant was
// negative).  Each field whose value changes is stored; returns whether any
// did.
// The fields go two at a time, their loads together (at in-range addresses: the
// point itself stands in for an axis that is not used); one after the other,
// each waited for the store of the one before.  192^3, order 2, eight fields:
// 100.9 -> 71.4 ms, one field 54.9 -> 54.4; 256^3, order 1: 121.6 -> 104, 63.0 -> 61.2.
// (Four at a time spill: 89.3 ms.)
__device__ __forceinline__ bool fmm_ext(const Update& U, const double i2[3], const ExtSet& X,
                                        long o, const long s[3]) {
  double w[3], den = 0;
  long a[3];
  bool used[3];
#pragma unroll
  for (int dir = 0; dir < 3; dir++) {
    const double g = U.second[dir] ? 1.5 * U.val - 2.0 * U.u1[dir] + 0.5 * U.u2[dir]
                                   : U.val - U.u1[dir];
    used[dir] = U.side[dir] >= 0;
    a[dir] = !used[dir] ? o : U.side[dir] == 1 ? o + s[dir] : o - s[dir];
    w[dir] = i2[dir] * g;
    if (used[dir]) den += w[dir];
  }
  bool changed = false;
  auto field = [&](int f, double old, double u0, double u1, double u2) {
    double num = 0;
    if (used[0]) num += w[0] * u0;
    if (used[1]) num += w[1] * u1;
    if (used[2]) num += w[2] * u2;
    const double v = num / den;
    if (__double_as_longlong(v) != __double_as_longlong(old)) {
      X.ext[f][o] = v;
      changed = true;
    }
  };
  int f = 0;
#pragma unroll 1
  for (; f + 1 < X.nf; f += 2) {
    const double *e = X.ext[f], *h = X.ext[f + 1];
    const double e0 = __ldcg(e + o), ea = __ldcg(e + a[0]), eb = __ldcg(e + a[1]),
                 ec = __ldcg(e + a[2]), h0 = __ldcg(h + o), ha = __ldcg(h + a[0]),
                 hb = __ldcg(h + a[1]), hc = __ldcg(h + a[2]);
    field(f, e0, ea, eb, ec);
    field(f + 1, h0, ha, hb, hc);
  }
  if (f < X.nf) {
    const double* e = X.ext[f];
    field(f, __ldcg(e + o), __ldcg(e + a[0]), __ldcg(e + a[1]), __ldcg(e + a[2]));
  }
  return changed;
}

// Device words of the solve.  The counts and minima gather over one pass and
// are read by every block after the barrier that ends it; three slots in
// turn, so that a slot is cleared a pass before its next use, when no block
// can still be reading it, and none adds to a slot that another reads.
struct Ctrl {
  int count[3];              // length of the active list of pass p: slot p % 3
  int pend_count[3];         // points pass p added to the pending list: slot p % 3
  unsigned long long minrej[3];   // bits of the smallest candidate among them
                                  // (times are >= 0),
  unsigned long long minkeep[3];  // and of those kept waiting: slot p % 3
  int pass;                  // result: passes run
  int done;                  // result: converged
  int error;                 // a barrier wait gave up
  alignas(128) unsigned arrived;  // blocks at the barrier, counted up for good
  alignas(128) unsigned released; // barriers passed
};

struct Lists {
  int* active;               // two lists of n points (by pass parity)
  int* stamp;                // pass that last queued a point
  int* pending;              // two lists of n points (by epoch parity)
  int* pend_stamp;           // epoch + 1 that last queued a point
  double2* vk;               // per point: value and key (kKeyFront, kKeyOutside)
  double* new_d;             // per slot of the active list beyond each thread's
  Time3* new_t;              //   first: the evaluated value (in the output
  unsigned char* new_f;      //   array), time and whether to store them
};

// grid coordinates of point o (the entry points limit grids to 2^31 - 1
// points, so 32-bit division is exact)
__device__ __forceinline__ void point_coords(long o, int nx, int ny, int c[3]) {
  const unsigned u = (unsigned)o, q = u / (unsigned)nx;
  c[0] = (int)(u - q * (unsigned)nx);
  c[1] = (int)(q % (unsigned)ny);
  c[2] = (int)(q / (unsigned)ny);
}

// the smallest of the warp's values (every lane takes part)
__device__ __forceinline__ unsigned long long warp_min(unsigned long long v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, off);
    v = o < v ? o : v;
  }
  return v;
}

// The points' pairs, and the first active list: the free points next to the
// front.
__global__ void k_fmm_seed(const double* d, const unsigned char* st, int nx, int ny, int nz,
                           Lists L, Ctrl* ctrl) {
  const long n = (long)nx * ny * nz;
  const long s[3] = {1L, (long)nx, (long)nx * ny};
  const int nn[3] = {nx, ny, nz};
  for (long o = blockIdx.x * (long)blockDim.x + threadIdx.x; o < n;
       o += (long)gridDim.x * blockDim.x) {
    L.vk[o] = make_double2(d[o], st[o] == kFront     ? kKeyFront
                                 : st[o] == kOutside ? kKeyOutside
                                                     : INFINITY);
    if (st[o] != kFree) continue;
    int c[3];
    point_coords(o, nx, ny, c);
    bool near = false;
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const int dir = q >> 1, sg = (q & 1) ? 1 : -1;
      const int c1 = c[dir] + sg;
      if (c1 >= 0 && c1 < nn[dir] && st[o + sg * s[dir]] == kFront) near = true;
    }
    if (near) {
      L.stamp[o] = 1;
      L.active[atomicAdd(&ctrl->count[0], 1)] = (int)o;
    }
  }
}

// Once the queued points fall to 1/kTailFraction of the threshold step's
// largest pass, the threshold moves on.  Each step has a burst of large
// passes and then a long tail of small ones as the last revisions settle;
// the threshold need not wait for that tail (the fixed point does not
// depend on when T moves, only the amount of revision does).  4 against 8:
// 442 passes for 493 (128x112x120, order 1), the points up by a sixth, the
// time down by 6 to 14 % over the sizes tried.
constexpr int kTailFraction = 4;

// Threads of a block of k_fmm_march, one block per SM (or of the one
// cluster): 128 registers a thread, 168 at order 2 over the GPU (with 512
// threads there 17.4 ms for 16.7 at 128x112x120; in the cluster 6.2 for 6.5 at
// 301x237).
__host__ __device__ constexpr int march_threads(int order, bool cluster) {
  return order == 1 || cluster ? 512 : 384;
}
constexpr int kClusterBlocks = 8;

// Whether the march runs on one cluster: its barrier takes less than that of a
// cooperative launch over the GPU, but its lists wait for the threads of 8 SMs.
// The lists grow with the size of the fronts, some n^(1/2) on a plane and n^(2/3)
// in space, and a point's evaluation takes about twice as long at second order,
// a ninth longer with each field and a fifth less for the Eikonal solver.  Both
// sides measured, in ms, cluster and GPU (six spheres, threshold steps of 6 cells):
//   order 1:           362^2 6.6, 7.5    512^2 12.6, 12.2   1500^2  91, 48
//   order 1, 8 fields: 181^2 3.9, 4.4    362^2 11.4, 10.4   1500^2 175, 67
//   order 2:           181^2 3.8, 4.0    256^2  6.5, 6.3    1500^2 156, 58
//   order 2, 8 fields: 128^2 3.7, 3.8    181^2  6.5, 6.2    1500^2 295, 97
//   Eikonal:           362^2 6.1, 6.8    724^2 18.4, 16.5   1500^2  76, 42
//   Eikonal, order 2:  256^2 5.6, 5.5    362^2  9.7, 8.5    1500^2 132, 52
//   24^3: order 1 0.67, 0.72, order 2 1.5, 1.2; 32^3: 1.2, 1.0 and 2.8, 1.7
// (The line was 1,536 cells on a plane's shorter side for every solve: 1500^2 had
// become slower than with two kernels a pass, 137 ms at order 2.)
bool march_on_cluster(const int* dims, int order, int fields, bool eikonal) {
  const double n = (double)dims[0] * dims[1] * dims[2];
  const bool flat = dims[0] == 1 || dims[1] == 1 || dims[2] == 1;
  const double front = 2.0 * (flat ? sqrt(n) : cbrt(n * n));
  const double line = (order == 1 ? 960.0 : 440.0) * (eikonal ? 1.25 : 1.0);
  return front * (1.0 + fields / 9.0) <= line;
}

constexpr unsigned long long kInfBits = 0x7ff0000000000000ULL;   // +infinity

// polls of a grid barrier before it gives up (seconds)
constexpr int kBarrierPolls = 1 << 24;

// Every block of the march has arrived (and its writes are visible) when
// this returns.  One cluster: the hardware barrier.  Else the blocks of a
// cooperative launch count themselves in and wait for the last one's word;
// a wait that gives up sets ctrl->error and returns false to every thread.
template <bool CLUSTER>
__device__ __forceinline__ bool march_barrier(Ctrl* ctrl, unsigned& gen, int* s_ok) {
  if constexpr (CLUSTER) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  } else {
    gen++;
    __syncthreads();
    if (threadIdx.x == 0) {
      int ok = 1;
      __threadfence();
      if (atomicAdd(&ctrl->arrived, 1u) == gen * gridDim.x - 1) {
        __threadfence();
        *(volatile unsigned*)&ctrl->released = gen;
      } else {
        int polls = 0;
        while (*(volatile unsigned*)&ctrl->released < gen)
          if (++polls == kBarrierPolls) {
            *(volatile int*)&ctrl->error = 1;
            ok = 0;
            break;
          }
      }
      __threadfence();
      *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
  }
}

// *p exchanged with v where the predicate holds, and the old value; v elsewhere
__device__ __forceinline__ int exch_if(unsigned pred, int* p, int v) {
  int old;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.b32 %0, %2;\n\t"
      "@q atom.global.exch.b32 %0, [%1], %2;\n\t}"
      : "=&r"(old)
      : "l"(p), "r"(v), "r"(pred)
      : "memory");
  return old;
}

// This thread's points go to positions of two lists, `mine` (0..12) and
// `mine2` (0 or 1) of them: the block reserves its room with one addition to
// each list's length (same-address atomics of every warp of the grid took
// longer than the evaluation).  Returns the thread's first position in each.
// Every thread of the block takes part.
struct Room {
  int warp_at[2][16];
  int base[2];
};
__device__ __forceinline__ int2 reserve(int mine, int mine2, int* count, int* count2, Room* r) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int upto = mine;
#pragma unroll
  for (int sh = 1; sh < 32; sh <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, upto, sh);
    if (lane >= sh) upto += v;
  }
  const unsigned ones = __ballot_sync(0xffffffffu, mine2 != 0);
  if (lane == 31) {
    r->warp_at[0][wid] = upto;
    r->warp_at[1][wid] = __popc(ones);
  }
  __syncthreads();
  if (wid == 0) {
    // lanes 0..15: the first list's warps, 16..31: the second's
    const int half = lane >> 4, w = lane & 15;
    int n = w < nw ? r->warp_at[half][w] : 0;
    const int own = n;
#pragma unroll
    for (int sh = 1; sh < 16; sh <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, n, sh, 16);
      if (w >= sh) n += v;
    }
    if (w < nw) r->warp_at[half][w] = n - own;
    if (w == 15) r->base[half] = n ? atomicAdd(half ? count2 : count, n) : 0;
  }
  __syncthreads();
  const int2 at = make_int2(r->base[0] + r->warp_at[0][wid] + upto - mine,
                            r->base[1] + r->warp_at[1][wid] +
                                __popc(ones & ((1u << lane) - 1u)));
  __syncthreads();   // the words are free for the next call
  return at;
}

// The whole march.  A pass p over its active list:
//   - each point's value and time from the values before the pass (evaluated
//     in place, while others change, a half-written neighbour can sustain
//     an oscillation that sequential or synchronous sweeps never enter);
//     rejected points join the pending list, the readers of a changed point
//     the list of pass p + 1 (stamped p + 2);
//   - after a threshold advance, the pending points of the last epoch that
//     the new threshold reaches join that list too, the others wait in this
//     epoch's pending list;
//   - barrier; the changes are stored; barrier;
//   - every block draws the same conclusion from the counts: the pass done,
//     the threshold moved, or the march ended (nothing queued or waiting).
// The passes are a chain of memory round trips over short lists (a few
// thousand to some ten thousand points), so their number times the latency of
// one is the time.  As two kernels a pass in a replayed graph, with a third
// of the time between kernels, a pass took 17 to 20 us (128x112x120, order 2:
// 24.9 ms a call from host arrays; 301x237, two extension fields: 11.9 ms).
// Here the readers are queued by the thread that found the change, beside
// the evaluation, a thread keeps its first slot's result in registers, the
// stamps of a point's readers are exchanged together, the warps of a short
// list are spread over the SMs, and a neighbour is one 16-byte load (value,
// time and status apart were a third more loads each, scattered over as many
// sectors: 35 us a pass at 68,000 points, 10.5 at 1,700).  9 to 14 us a pass
// where the lists are short (half of it the evaluation, the rest the two
// barriers and the queue), 31 at 68,000 points.
// Short lists run on one cluster of 8 SMs, whose barrier is a hardware one
// (march_on_cluster).
// SOLVE: the distance function alone, with extension fields (whose values cost
// registers that the others keep), or the Eikonal solver.
enum { kSolveDistance, kSolveExtension, kSolveEikonal };
template <int ORDER, int SOLVE, bool CLUSTER>
__global__ void __launch_bounds__(march_threads(ORDER, CLUSTER), 1)
k_fmm_march(double2* tm, int nx, int ny, int nz, double i2x, double i2y, double i2z, Lists L,
            Ctrl* ctrl, ExtSet X, Eik E, double delta, int max_passes) {
  constexpr bool EIK = SOLVE == kSolveEikonal;
  constexpr int kReaders = 6 * ORDER;
  __shared__ Room room;
  __shared__ unsigned long long s_min[2];
  __shared__ struct {
    int count, waiting, filter, ep, advance, done;
    double T;
  } c_;
  __shared__ int s_ok;
  const long n = (long)nx * ny * nz;
  double2* const vk = L.vk;
  const int lane = threadIdx.x & 31;
  const int nb = (int)gridDim.x, bid = (int)blockIdx.x;
  const int total = nb * (int)blockDim.x;
  // slot of a round: warps go over the blocks first
  const int slot = (((int)threadIdx.x >> 5) * nb + bid) * 32 + lane;
  const double i2[3] = {i2x, i2y, i2z};
  const int nn[3] = {nx, ny, nz};
  const long s[3] = {1L, (long)nx, (long)nx * ny};
  unsigned gen = 0;
  // thread 0: the largest queue of the threshold step, its smallest candidate
  int peak = 0;
  unsigned long long smallest = kInfBits;
  if (threadIdx.x == 0) {
    c_.count = __ldcg(&ctrl->count[0]);
    c_.T = delta;
    c_.ep = c_.waiting = c_.filter = c_.advance = c_.done = 0;
    s_min[0] = s_min[1] = kInfBits;
  }
  __syncthreads();
  int pass = 0;
  for (; pass < max_passes; pass++) {
    const int count = c_.count, ep = c_.ep;
    const double T = c_.T;
    const int* cur = L.active + (pass & 1) * n;
    int* next = L.active + ((pass + 1) & 1) * n;
    int* next_count = &ctrl->count[(pass + 1) % 3];
    int* pend = L.pending + (ep & 1) * n + c_.waiting;
    int* pend_count = &ctrl->pend_count[pass % 3];
    if (bid == 0 && threadIdx.x == 0) {
      ctrl->count[(pass + 2) % 3] = 0;
      ctrl->pend_count[(pass + 1) % 3] = 0;
      ctrl->minrej[(pass + 1) % 3] = ctrl->minkeep[(pass + 1) % 3] = kInfBits;
    }
    unsigned long long minrej = kInfBits, minkeep = kInfBits;
    // the first slot's result
    bool f_first = false;
    int o_first = 0;
    double d_first = 0;
    Time3 t_first{0, 0, 0};
    for (int base = 0; base + bid * 32 < count; base += total) {
      const int w = base + slot;
      unsigned won = 0;
      bool wait = false;
      long o = 0;
      if (w < count) {
        o = __ldcg(cur + w);
        // only free points are ever queued; the value and time of the
        // point itself are loaded beside its stencil
        const double2 self = __ldcg(vk + o);
        const double old = self.x, told_b = __ldcg(&tm[o].x);
        int c[3];
        point_coords(o, nx, ny, c);
        Update U;
        unsigned cand;
        int reached = fmm_point_fast<ORDER, EIK>(vk, tm, o, c, nn, s, i2, E, U, cand);
        if (reached < 0) {
          Update slow;
          reached = fmm_point<ORDER, EIK>(vk, tm, o, c[0], c[1], c[2], nx, ny, nz, i2x, i2y, i2z,
                                          E, &slow);
          U = slow;
        }
        double val = U.val;
        Time3 tv = U.t;
        bool ext_changed = false;
        if (!reached) {
          // no neighbour is reached (any more): no update, the point is unreached
          val = copysign(INFINITY, old);
          tv = Time3{INFINITY, INFINITY, INFINITY};
        } else if (!(tv.a <= T)) {
          // accepted after the threshold: a candidate only, waiting for T
          val = copysign(INFINITY, old);
          wait = atomicExch(L.pend_stamp + o, ep + 1) != ep + 1;
          const unsigned long long bits = __double_as_longlong(tv.a);
          minrej = bits < minrej ? bits : minrej;
        } else if (SOLVE == kSolveExtension) {
          ext_changed = fmm_ext(U, i2, X, o, s);
        }
        // (the third level counts where the second does)
        const bool store = ext_changed || !(val == old && tv.a == self.y && tv.b == told_b &&
                                            (tv.b == -1.0 || tv.c == __ldcg(&tm[o].y)));
        if (base == 0) {
          f_first = store;
          o_first = (int)o;
          d_first = val;
          t_first = tv;
        } else {
          L.new_f[w] = store;
          L.new_d[w] = val;
          L.new_t[w] = tv;
        }
        // the free points whose stencil reads this one, where the change is
        // visible: the value is finite before or after, or a field changed
        if (store && (ext_changed || fabs(old) <= DBL_MAX || fabs(val) <= DBL_MAX)) {
          // the exchanges go out together: predicated, without branches
          int was[kReaders];
#pragma unroll
          for (int k = 0; k < kReaders; k++)
            was[k] = exch_if(cand >> k & 1, L.stamp + nb_index(o, s, k / ORDER, k % ORDER + 1),
                             pass + 2);
#pragma unroll
          for (int k = 0; k < kReaders; k++)
            if (was[k] != pass + 2) won |= 1u << k;
        }
      }
      const int2 at = reserve(__popc(won), wait, next_count, pend_count, &room);
      if (wait) pend[at.y] = (int)o;
      int pos = at.x;
#pragma unroll
      for (int k = 0; k < kReaders; k++)
        if (won >> k & 1) next[pos++] = (int)nb_index(o, s, k / ORDER, k % ORDER + 1);
    }
    // the pending points of the last epoch after a threshold advance.  Values
    // and times do not change before the barrier, so the test reads them as
    // the pass does.
    const int filter = c_.advance ? c_.filter : 0;
    const int* src = L.pending + ((ep - 1) & 1) * n;
    for (int base = 0; base + bid * 32 < filter; base += total) {
      const int w = base + slot;
      bool go = false, wait = false;
      int o = 0;
      if (w < filter) {
        o = __ldcg(src + w);
        const double2 self = __ldcg(vk + o);
        const double t = self.y;
        if (!(fabs(self.x) <= DBL_MAX)) {   // not reached since
          if (t <= T) {
            go = atomicExch(L.stamp + o, pass + 2) != pass + 2;
          } else if (t < INFINITY) {
            wait = atomicExch(L.pend_stamp + o, ep + 1) != ep + 1;
            const unsigned long long bits = __double_as_longlong(t);
            minkeep = bits < minkeep ? bits : minkeep;
          }
        }
      }
      const int2 at = reserve(go, wait, next_count, pend_count, &room);
      if (go) next[at.x] = o;
      if (wait) pend[at.y] = o;
    }
    minrej = warp_min(minrej);
    minkeep = warp_min(minkeep);
    if (lane == 0) {
      if (minrej != kInfBits) atomicMin(&s_min[0], minrej);
      if (minkeep != kInfBits) atomicMin(&s_min[1], minkeep);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (s_min[0] != kInfBits) atomicMin(&ctrl->minrej[pass % 3], s_min[0]);
      if (s_min[1] != kInfBits) atomicMin(&ctrl->minkeep[pass % 3], s_min[1]);
      s_min[0] = s_min[1] = kInfBits;
    }
    if (!march_barrier<CLUSTER>(ctrl, gen, &s_ok)) return;
    if (f_first) {
      vk[o_first] = make_double2(d_first, t_first.a);
      tm[o_first] = make_double2(t_first.b, t_first.c);
    }
    for (int w = slot + total; w < count; w += total)
      if (L.new_f[w]) {
        const int o = __ldcg(cur + w);
        const Time3 t = L.new_t[w];
        vk[o] = make_double2(L.new_d[w], t.a);
        tm[o] = make_double2(t.b, t.c);
      }
    if (!march_barrier<CLUSTER>(ctrl, gen, &s_ok)) return;
    // thread 0 of each block: the threshold control, from the same words in
    // every block
    if (threadIdx.x == 0) {
      const int queued = __ldcg(next_count), np = c_.waiting + __ldcg(pend_count);
      const unsigned long long rej = __ldcg(&ctrl->minrej[pass % 3]),
                               keep = __ldcg(&ctrl->minkeep[pass % 3]);
      smallest = rej < smallest ? rej : smallest;
      smallest = keep < smallest ? keep : smallest;
      peak = queued > peak ? queued : peak;
      c_.waiting = np;
      c_.advance = 0;
      if ((long)queued * kTailFraction <= peak) {
        if (np == 0) {
          if (queued == 0) c_.done = 1;
        } else {
          const double lo = __longlong_as_double((long long)smallest);
          const double step = T + delta;
          c_.T = lo > step ? lo : step;
          c_.advance = 1;
          c_.filter = np;
          c_.waiting = 0;
          c_.ep = ep + 1;
          peak = queued;
          smallest = kInfBits;
        }
      }
      c_.count = queued;
    }
    __syncthreads();
    if (c_.done) {
      pass++;
      break;
    }
  }
  if (bid == 0 && threadIdx.x == 0) {
    ctrl->pass = pass;
    ctrl->done = c_.done;
  }
}

// The values of all points (the march used the output array); free points no
// front reached take the reference's default value -1 (distance and extension
// fields), or the Eikonal solver's input
__global__ void k_fmm_finish(double* d, const double2* vk, const unsigned char* st, long n,
                             ExtSet X, const double* phi0) {
  for (long o = blockIdx.x * (long)blockDim.x + threadIdx.x; o < n;
       o += (long)gridDim.x * blockDim.x) {
    const double v = vk[o].x;
    if (st[o] != kFree || fabs(v) <= DBL_MAX) {
      d[o] = v;
      continue;
    }
    d[o] = phi0 ? phi0[o] : -1.0;
    for (int f = 0; f < X.nf; f++) X.ext[f][o] = -1.0;
  }
}

// One solve on device arrays: the distance function and up to kMaxFields
// extension fields (X.nf may be 0), or with E.speed the Eikonal solution
// for the boundary data E.phi0 (dp unused).
bool solve_device(double* dd, const double* dp, const double* dm, const ExtSet& X,
                  const Eik& E, int order, const int* grid_dims, const double* dx,
                  int* passes_out, const char* R, cudaStream_t st) {
  const int nx = grid_dims[0], ny = grid_dims[1], nz = grid_dims[2];
  const long n = (long)nx * ny * nz;
  const double hmin = fmin(dx[0], fmin(dx[1], dx[2]));
  // a bound on the passes for inputs without a fixed point (NaN): the
  // threshold crosses the grid in at most (diagonal / delta) steps of a
  // few passes each
  const long max_passes = 4096 + 32L * (nx + ny + nz);
  unsigned char* status = nullptr;
  double2* tm = nullptr;
  // points of a typical list: two per point of the grid's largest cross-section
  const int longest = nx > ny ? (nx > nz ? nx : nz) : (ny > nz ? ny : nz);
  const long band = 2 * n / longest;
  Lists L{};
  L.new_d = dd;   // the output, which k_fmm_finish writes
  Ctrl* ctrl = nullptr;
  const size_t un = (size_t)n;
  bool ok = cuda_ok(pool_alloc((void**)&status, un, st), R) &&
            cuda_ok(pool_alloc((void**)&tm, un * sizeof(double2), st), R) &&
            cuda_ok(pool_alloc((void**)&L.active, 2 * un * sizeof(int), st), R) &&
            cuda_ok(pool_alloc((void**)&L.pending, 2 * un * sizeof(int), st), R) &&
            cuda_ok(pool_alloc((void**)&L.stamp, un * sizeof(int), st), R) &&
            cuda_ok(pool_alloc((void**)&L.pend_stamp, un * sizeof(int), st), R) &&
            cuda_ok(pool_alloc((void**)&L.vk, un * sizeof(double2), st), R) &&
            cuda_ok(pool_alloc((void**)&L.new_t, un * sizeof(Time3), st), R) &&
            cuda_ok(pool_alloc((void**)&L.new_f, un, st), R) &&
            cuda_ok(pool_alloc((void**)&ctrl, sizeof(Ctrl), st), R);
  Ctrl h_ctrl{};
  for (int q = 0; q < 3; q++) h_ctrl.minrej[q] = h_ctrl.minkeep[q] = kInfBits;
  int sms = 148;
  {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess)
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const int elem_blocks = (int)((n + 255) / 256 < 8 * sms ? (n + 255) / 256 : 8 * sms);
  if (ok) {
    ok = cuda_ok(cudaMemsetAsync(L.stamp, 0, un * sizeof(int), st), R) &&
         cuda_ok(cudaMemsetAsync(L.pend_stamp, 0, un * sizeof(int), st), R) &&
         cuda_ok(cudaMemcpyAsync(ctrl, &h_ctrl, sizeof(Ctrl), cudaMemcpyHostToDevice, st), R);
  }
  if (ok) {
    const dim3 blk(32, 4, 1);
    const dim3 grid3((nx + 31) / 32, (ny + 3) / 4, nz < 65535 ? nz : 65535);
    if (E.speed)
      k_eik_front<<<elem_blocks, 256, 0, st>>>(dd, tm, status, E.phi0, E.speed, dm, n);
    else
      k_fmm_front<<<grid3, blk, 0, st>>>(dd, tm, status, dp, dm, nx, ny, nz, dx[0], dx[1],
                                         dx[2], X);
    k_fmm_seed<<<elem_blocks, 256, 0, st>>>(dd, status, nx, ny, nz, L, ctrl);
    launch_counter() += 2;
    ok = cuda_ok(cudaGetLastError(), R);
  }
  // 1/dx, squared (:1077-1078)
  double i2[3];
  for (int q = 0; q < 3; q++) {
    i2[q] = 1 / dx[q];
    i2[q] *= i2[q];
  }
  // One cluster while its 8 SMs hold the lists, else one block per SM of a
  // cooperative launch; and the threshold's step
  const bool cluster = march_on_cluster(grid_dims, order, X.nf, E.speed != nullptr);
  const bool small = cluster || 4 * band <= (long)sms * march_threads(order, false);
  const double delta = (small ? kDeltaCellsSmall : kDeltaCells) * hmin;
  // (passes in whole batches of 32)
  int passes = (int)((max_passes + 31) / 32 * 32);
  if (ok) {
#define MARCH(O, K) \
  (cluster ? (const void*)k_fmm_march<O, K, true> : (const void*)k_fmm_march<O, K, false>)
#define SOLVE(O)                            \
  (E.speed ? MARCH(O, kSolveEikonal)        \
           : X.nf ? MARCH(O, kSolveExtension) : MARCH(O, kSolveDistance))
    const void* fn = order == 1 ? SOLVE(1) : SOLVE(2);
#undef SOLVE
#undef MARCH
    ExtSet xs = X;
    Eik es = E;
    double step = delta;
    int mx = nx, my = ny, mz = nz;
    void* args[] = {&tm, &mx, &my, &mz, &i2[0], &i2[1], &i2[2], &L, &ctrl, &xs, &es, &step,
                    &passes};
    cudaLaunchAttribute at{};
    at.id = cluster ? cudaLaunchAttributeClusterDimension : cudaLaunchAttributeCooperative;
    if (cluster) {
      at.val.clusterDim.x = kClusterBlocks;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
    } else {
      at.val.cooperative = 1;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cluster ? kClusterBlocks : sms);
    cfg.blockDim = dim3(march_threads(order, cluster));
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    ok = cuda_ok(cudaLaunchKernelExC(&cfg, fn, args), R);
    ++launch_counter();
    ok = ok &&
         cuda_ok(cudaMemcpyAsync(&h_ctrl, ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, st), R) &&
         cuda_ok(cudaStreamSynchronize(st), R);
    if (ok && h_ctrl.error) {
      set_error(LSMGPU_ERR_DEVICE, std::string(R) + ": a wait between blocks gave up");
      ok = false;
    } else if (ok && !h_ctrl.done) {
      set_error(LSMGPU_ERR_INVALID_VALUE, std::string(R) + ": no convergence (NaN in phi?)");
      ok = false;
    }
  }
  if (ok) {
    k_fmm_finish<<<elem_blocks, 256, 0, st>>>(dd, L.vk, status, n, X, E.phi0);
    ++launch_counter();
    ok = cuda_ok(cudaGetLastError(), R);
  }
  for (void* q : {(void*)status, (void*)tm, (void*)L.active, (void*)L.pending,
                  (void*)L.stamp, (void*)L.pend_stamp, (void*)L.vk, (void*)L.new_t,
                  (void*)L.new_f, (void*)ctrl})
    if (q) cudaFreeAsync(q, st);
  if (passes_out) *passes_out = h_ctrl.pass;
  return ok;
}

// computeExtensionFields3d / computeDistanceFunction3d on host or device
// arrays: argument checks, staging, and one solve per group of kMaxFields
// fields (each solve recomputes the same distance function).
int extension3d(double* distance, double** ext, const double* phi, const double* mask,
                double* const* src, const double* emask, int nf, int order,
                const int* grid_dims, const double* dx, int* passes_out, const char* R) {
  clear_error();
  if (!distance || !phi || !grid_dims || !dx || (nf > 0 && (!ext || !src))) {
    set_error(LSMGPU_ERR_NULL_POINTER, std::string(R) + ": null argument");
    return LSMGPU_ERR_NULL_POINTER;
  }
  for (int k = 0; k < nf; k++)
    if (!ext[k] || !src[k]) {
      set_error(LSMGPU_ERR_NULL_POINTER, std::string(R) + ": null field pointer");
      return LSMGPU_ERR_NULL_POINTER;
    }
  if (nf < 0) {
    set_error(LSMGPU_ERR_INVALID_VALUE, std::string(R) + ": negative field count");
    return LSMGPU_ERR_INVALID_VALUE;
  }
  if (order != 1 && order != 2) {
    set_error(LSMGPU_ERR_INVALID_VALUE, std::string(R) + ": order is 1 or 2");
    return LSMGPU_ERR_INVALID_VALUE;
  }
  const int nx = grid_dims[0], ny = grid_dims[1], nz = grid_dims[2];
  if (nx < 1 || ny < 1 || nz < 1) {
    set_error(LSMGPU_ERR_INVALID_BOX, std::string(R) + ": empty grid");
    return LSMGPU_ERR_INVALID_BOX;
  }
  if (!(dx[0] > 0) || !(dx[1] > 0) || !(dx[2] > 0) || !(dx[0] < INFINITY) ||
      !(dx[1] < INFINITY) || !(dx[2] < INFINITY)) {
    set_error(LSMGPU_ERR_INVALID_VALUE, std::string(R) + ": dx must be positive and finite");
    return LSMGPU_ERR_INVALID_VALUE;
  }
  if ((long)nx * ny * nz > 0x7fffffffL) {
    set_error(LSMGPU_ERR_INVALID_BOX, std::string(R) + ": more than 2^31 - 1 points");
    return LSMGPU_ERR_INVALID_BOX;
  }
  cudaStream_t st = cur_stream();
  Staging stg(st);
  const Box b{{0, 0, 0}, {nx, ny, nz}};
  double* dd = (double*)stg.add(distance, b, 8, kOutFull, "distance_function", R);
  const double* dp = dd ? (const double*)stg.add(phi, b, 8, kIn, "phi", R) : nullptr;
  const double* dm = nullptr;
  if (dp && mask) dm = (const double*)stg.add(mask, b, 8, kIn, "mask", R);
  const double* dem = nullptr;
  if (dp && emask) dem = (const double*)stg.add(emask, b, 8, kIn, "extension_mask", R);
  if (!dd || !dp || (mask && !dm) || (emask && !dem)) return lsmgpu_peek_last_error();
  int group = 0;
  do {
    ExtSet X{};
    X.emask = dem;
    X.nf = nf - group < kMaxFields ? nf - group : kMaxFields;
    for (int k = 0; k < X.nf; k++) {
      X.ext[k] = (double*)stg.add(ext[group + k], b, 8, kOutFull, "extension_field", R);
      X.src[k] = X.ext[k] ? (const double*)stg.add(src[group + k], b, 8, kIn, "source_field",
                                                   R)
                          : nullptr;
      if (!X.ext[k] || !X.src[k]) return lsmgpu_peek_last_error();
    }
    if (!solve_device(dd, dp, dm, X, Eik{nullptr, nullptr}, order, grid_dims, dx, passes_out,
                      R, st))
      return lsmgpu_peek_last_error() ? lsmgpu_peek_last_error() : LSMGPU_ERR_CUDA;
    group += X.nf;
  } while (group < nf);
  return stg.finish(R) ? LSMGPU_SUCCESS : LSMGPU_ERR_CUDA;
}

// solveEikonalEquation3d on host or device arrays: phi holds the boundary
// data on input and the solution on output.
int eikonal3d(double* phi, const double* speed, const double* mask, int order,
              const int* grid_dims, const double* dx, int* passes_out, const char* R) {
  clear_error();
  if (!phi || !speed || !grid_dims || !dx) {
    set_error(LSMGPU_ERR_NULL_POINTER, std::string(R) + ": null argument");
    return LSMGPU_ERR_NULL_POINTER;
  }
  if (order != 1 && order != 2) {
    set_error(LSMGPU_ERR_INVALID_VALUE, std::string(R) + ": order is 1 or 2");
    return LSMGPU_ERR_INVALID_VALUE;
  }
  const int nx = grid_dims[0], ny = grid_dims[1], nz = grid_dims[2];
  if (nx < 1 || ny < 1 || nz < 1) {
    set_error(LSMGPU_ERR_INVALID_BOX, std::string(R) + ": empty grid");
    return LSMGPU_ERR_INVALID_BOX;
  }
  if (!(dx[0] > 0) || !(dx[1] > 0) || !(dx[2] > 0) || !(dx[0] < INFINITY) ||
      !(dx[1] < INFINITY) || !(dx[2] < INFINITY)) {
    set_error(LSMGPU_ERR_INVALID_VALUE, std::string(R) + ": dx must be positive and finite");
    return LSMGPU_ERR_INVALID_VALUE;
  }
  const long n = (long)nx * ny * nz;
  if (n > 0x7fffffffL) {
    set_error(LSMGPU_ERR_INVALID_BOX, std::string(R) + ": more than 2^31 - 1 points");
    return LSMGPU_ERR_INVALID_BOX;
  }
  cudaStream_t st = cur_stream();
  Staging stg(st);
  const Box b{{0, 0, 0}, {nx, ny, nz}};
  double* dd = (double*)stg.add(phi, b, 8, kInOut, "phi", R);
  const double* df = dd ? (const double*)stg.add(speed, b, 8, kIn, "speed", R) : nullptr;
  const double* dm = nullptr;
  if (df && mask) dm = (const double*)stg.add(mask, b, 8, kIn, "mask", R);
  if (!dd || !df || (mask && !dm)) return lsmgpu_peek_last_error();
  double* phi0 = nullptr;
  bool ok = cuda_ok(pool_alloc((void**)&phi0, (size_t)n * sizeof(double), st), R) &&
            cuda_ok(cudaMemcpyAsync(phi0, dd, (size_t)n * sizeof(double),
                                    cudaMemcpyDeviceToDevice, st), R);
  ok = ok && solve_device(dd, nullptr, dm, ExtSet{}, Eik{df, phi0}, order, grid_dims, dx,
                          passes_out, R, st);
  if (phi0) cudaFreeAsync(phi0, st);
  if (!ok) return lsmgpu_peek_last_error() ? lsmgpu_peek_last_error() : LSMGPU_ERR_CUDA;
  return stg.finish(R) ? LSMGPU_SUCCESS : LSMGPU_ERR_CUDA;
}

}  // namespace

extern "C" {

// lsm_fast_marching_method.h:386-392: 0 on success, 2 for an order other
// than 1 or 2 (LSM_FMM_ERR_INVALID_SPATIAL_DISCRETIZATION_ORDER), -1 for any
// other failure (the lsmgpu error is recorded)
int computeDistanceFunction3d(double* distance_function, double* phi, double* mask,
                              int spatial_discretization_order, int* grid_dims,
                              double* dx) {
  if (spatial_discretization_order != 1 && spatial_discretization_order != 2) return 2;
  const int rc = extension3d(distance_function, nullptr, phi, mask, nullptr, nullptr, 0,
                             spatial_discretization_order, grid_dims, dx, nullptr,
                             "computeDistanceFunction3d");
  return rc == LSMGPU_SUCCESS ? 0 : -1;
}

// lsm_fast_marching_method.h:331-341, the same return codes
int computeExtensionFields3d(double* distance_function, double** extension_fields,
                             double* phi, double* mask, double** source_fields,
                             double* extension_mask, int num_extension_fields,
                             int spatial_discretization_order, int* grid_dims, double* dx) {
  if (spatial_discretization_order != 1 && spatial_discretization_order != 2) return 2;
  const int rc = extension3d(distance_function, extension_fields, phi, mask, source_fields,
                             extension_mask, num_extension_fields,
                             spatial_discretization_order, grid_dims, dx, nullptr,
                             "computeExtensionFields3d");
  return rc == LSMGPU_SUCCESS ? 0 : -1;
}

int lsmgpu_distance_function3d(double* distance_function, const double* phi,
                               const double* mask, int order, const int* grid_dims,
                               const double* dx, int* passes) {
  return extension3d(distance_function, nullptr, phi, mask, nullptr, nullptr, 0, order,
                     grid_dims, dx, passes, "lsmgpu_distance_function3d");
}

int lsmgpu_extension_fields3d(double* distance_function, double** extension_fields,
                              const double* phi, const double* mask,
                              double* const* source_fields, const double* extension_mask,
                              int num_extension_fields, int order, const int* grid_dims,
                              const double* dx, int* passes) {
  return extension3d(distance_function, extension_fields, phi, mask, source_fields,
                     extension_mask, num_extension_fields, order, grid_dims, dx, passes,
                     "lsmgpu_extension_fields3d");
}

// lsm_fast_marching_method.h:463-469, the same return codes
int solveEikonalEquation3d(double* phi, double* speed, double* mask,
                           int spatial_discretization_order, int* grid_dims, double* dx) {
  if (spatial_discretization_order != 1 && spatial_discretization_order != 2) return 2;
  const int rc = eikonal3d(phi, speed, mask, spatial_discretization_order, grid_dims, dx,
                           nullptr, "solveEikonalEquation3d");
  return rc == LSMGPU_SUCCESS ? 0 : -1;
}

int lsmgpu_eikonal3d(double* phi, const double* speed, const double* mask, int order,
                     const int* grid_dims, const double* dx, int* passes) {
  return eikonal3d(phi, speed, mask, order, grid_dims, dx, passes, "lsmgpu_eikonal3d");
}

// The 2D forms (lsm_fast_marching_method.h:124-134, 179-185, 256-262): the
// 3D solve on a grid one plane thick, on which the reference's own 2D and 3D
// routines agree bit for bit.  grid_dims and dx hold x and y; the z spacing
// is taken as dx[0] (a single plane has no z neighbours, and the threshold
// step then still follows the smallest of dx and dy).  Null arguments pass
// through as null, so the 3D checks report them.
static void plane_grid(const int* grid_dims, const double* dx, int d3[3], double h3[3],
                       const int** pd, const double** ph) {
  *pd = nullptr;
  *ph = nullptr;
  if (grid_dims) {
    d3[0] = grid_dims[0];
    d3[1] = grid_dims[1];
    d3[2] = 1;
    *pd = d3;
  }
  if (dx) {
    h3[0] = dx[0];
    h3[1] = dx[1];
    h3[2] = dx[0];
    *ph = h3;
  }
}

int computeExtensionFields2d(double* distance_function, double** extension_fields,
                             double* phi, double* mask, double** source_fields,
                             double* extension_mask, int num_extension_fields,
                             int spatial_discretization_order, int* grid_dims, double* dx) {
  if (spatial_discretization_order != 1 && spatial_discretization_order != 2) return 2;
  int d3[3];
  double h3[3];
  const int* pd;
  const double* ph;
  plane_grid(grid_dims, dx, d3, h3, &pd, &ph);
  const int rc = extension3d(distance_function, extension_fields, phi, mask, source_fields,
                             extension_mask, num_extension_fields,
                             spatial_discretization_order, pd, ph, nullptr,
                             "computeExtensionFields2d");
  return rc == LSMGPU_SUCCESS ? 0 : -1;
}

int computeDistanceFunction2d(double* distance_function, double* phi, double* mask,
                              int spatial_discretization_order, int* grid_dims,
                              double* dx) {
  if (spatial_discretization_order != 1 && spatial_discretization_order != 2) return 2;
  int d3[3];
  double h3[3];
  const int* pd;
  const double* ph;
  plane_grid(grid_dims, dx, d3, h3, &pd, &ph);
  const int rc = extension3d(distance_function, nullptr, phi, mask, nullptr, nullptr, 0,
                             spatial_discretization_order, pd, ph, nullptr,
                             "computeDistanceFunction2d");
  return rc == LSMGPU_SUCCESS ? 0 : -1;
}

int solveEikonalEquation2d(double* phi, double* speed, double* mask,
                           int spatial_discretization_order, int* grid_dims, double* dx) {
  if (spatial_discretization_order != 1 && spatial_discretization_order != 2) return 2;
  int d3[3];
  double h3[3];
  const int* pd;
  const double* ph;
  plane_grid(grid_dims, dx, d3, h3, &pd, &ph);
  const int rc = eikonal3d(phi, speed, mask, spatial_discretization_order, pd, ph, nullptr,
                           "solveEikonalEquation2d");
  return rc == LSMGPU_SUCCESS ? 0 : -1;
}

}  // extern "C"
