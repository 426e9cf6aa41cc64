// "Walk" sweeps: the pruned DFD, VE-FD and decision DPs of a pair, block by block along its
// live band.
//
// At a level near its result a DP's live region is a thin band: on the uneven batch's pairs
// and on the 200,000-point pair it crosses an anti-diagonal in 1.5 to 10 cells and one or two
// blocks of 32 x 32 cells, whatever the curves' lengths.  The team strips (rfd_team.cuh) hand
// a row on from one 32-row strip to the next through L2 in 32-column chunks, which costs such
// a band about 11 us a strip.  Here one CTA walks the band instead:
//   warp 0 (propagator)    goes through the 32-row block rows in order and, in each, through
//                          the blocks that have a live input, left to right, one row at a time
//                          (lane = column): the row below is a short list of live 32-column
//                          chunks in shared memory, the column to the left one value per row;
//   warps 1..7 (helpers)   compute the block's cell values into a tile: a cheap test (point
//                          distance against the level plus a segment length) leaves the edges
//                          that can be live, which are listed and evaluated densely.  Values
//                          are kept in list order; per row, bit masks say which edges are
//                          listed and which came out live, so nothing is stored for the rest.
// While a block is swept the helpers fill the tile of the block most likely to be next (right
// when an edge of the last column is live, up otherwise).  The grid's rows run along the longer
// curve: a denser curve then moves the band up, which is the cheap direction of a row sweep.
//
// Exactness: a cell is skipped only when both its inputs are dead, an edge only when its value
// is certainly dead (empty interval, weight above the pruning bound), the rules of the pruned
// strips (rfd_device.cuh).  Live values are computed by the same functions from the same
// operands and combined by exact min, max and comparisons, so results are bit-identical, and
// the transposed grid gives the same values as for the strips (PairDesc::tr).
//
// Several CTAs share a long pair (a group): each walks a piece of the block rows.  Only the
// first knows the row its piece starts from, so the others start from everything that could
// be live there - every edge of that row with its free interval from its start, or its bare
// weight - which can only be more live, or smaller, than the truth.  A thin band forgets its
// start within a row or two: each piece is walked again from the end its predecessor came to,
// but only until a block row's list equals the one the first walk recorded there; from there on
// the first walk's is the true one.  For the min-max DPs "equals" is up to one constant: lists
// with values max(c, v) against v stay so for good (min and max distribute), and the constants
// of the pieces are combined at the end.  A piece that never meets its record hands its new
// end on to another round, so the outcome does not rest on the band being forgetful, and a
// piece that ends empty from everything that could be live ends the sweep (walk_sweep).  Once a
// sweep has found the band, the next ones start their pieces only near where it ran.
//
// A sweep whose band is not thin (list overflow, time against progress) gives up, and so does a
// phase past a share of the strips' time (walk_slow, walk_pair); the pair's phase then runs on the
// strips.
//
// What bounds it: the chain of a band's blocks.  A decision's block takes about 5,300 cycles (the
// rows 2,900, waiting for the tile 900, the next block's choice 500; a tile is ready 3,500 after
// its request), a VE-FD or DFD block with values about 10,000.  Against the strips, medians over
// twelve pairs of a size: search of 20,000 x 19,000 points 180 ms and 7.7 (4.1 to 16.3), 2,000 x 1,900
// 18.5 and 3.5; VE-FD and one decision of 200,000 x 200,000 95 and 3.8; bounds of 60,000 x 45,000
// points 35 and 2.1 to 5.0 where the walk holds, 26 to 32 where it gives the DFD up.
#pragma once

#include "rfd_device.cuh"
#include "rfd_filter.h"
#include "rfd_team.cuh"
#include "rfd_walk_cut.h"

namespace rfd {

constexpr int kWalkHelpers = 7;
constexpr int kWalkThreads = 32 * (kWalkHelpers + 1);
constexpr int kWalkCap = 24;         // live chunks of a block row's output list
constexpr double kDecDead = 4.0;     // dead decision value (live ones lie in [0, 1])
constexpr double kDecLive = 2.0;     // below: live

// Stage of a tile, in doubles: 33 points of each curve, then per row and per column the
// segment's A, 0.5/A and skip threshold.
constexpr int kWalkPts = 33 * 3;
constexpr int kWalkStage = 2 * kWalkPts + 6 * 32;
// Values of a tile: every edge's interval (decision) or weight (VE-FD), or every cell's point
// distance (DFD), in list order.
constexpr int kWalkVals = 2048;

// A block row's output list as recorded by the first walk of a piece (n < 0: too long to record),
// and the chunks lo .. hi of the list as last walked.
constexpr int kWalkRec = 4;
constexpr float kWalkClock = 1900.f;  // cycles a microsecond, about
struct WalkRecord {
  int n, lo, hi, pad;
  int j[kWalkRec];
  double v[kWalkRec][32];
};
struct WalkEnd {  // a piece's last list
  int n, pad;
  int j[kWalkCap];
  double v[kWalkCap][32];
};
// What a member reports at the end of a round: constant and result of its piece, whether its end
// changed in the round, which copy of the end is current (0: the first walk's, 1 or 2), whether
// it is empty; part: the first walk did not start from everything, or lost something on the way;
// skip: the piece has no rows (its members' neighbours are each other's).
struct WalkStat {
  double c, res;
  int changed, which, empty, part, gave_up, skip;
};
// WalkStat::gave_up: the piece ends the phase; past the phase's deadline; the first walk, from what
// could be live, was given up (the piece is left to the rounds).
constexpr int kGaveUp = 1, kLate = 2, kCrowded = 4;
// Points 32 J .. 32 J + 32 of a curve within rad of the centre (rad infinite: no bound).
struct WalkBall {
  double x[3], rad;
};

constexpr int kScan = -3;  // request word: the columns that can be live in the row below a piece

struct WalkShared {
  unsigned long long full[2];  // helpers -> propagator: tile ready
  unsigned long long req[2];   // propagator -> helpers: tile requested
  int req_i[2], req_j[2];      // block row (kStop: leave) and column
  int cancel[2];               // the speculative tile is not needed
  int cnt[2];                  // edges listed
  int scan_to;                 // list a scan fills
  PairDesc pd;                 // the running sweep's grid
  const double2 *seg_r, *seg_c;  // (|segment|^2, 0.5 / that) of the rows' and columns' segments,
  int step_r, step_c;            // every step-th double2
  int kind, flat, filter, mat;
  double level, rad;           // pruning bound U or radius^2, and its root
  unsigned long long cells, cells64;
  uint4 mask[2][32];           // per row: listed right, listed top, live right, live top edges
  uint4 risk[2][32];           // per row: right edges that end before 1, that start after 0, top
                               // edges that end before 1
  uint4 row_bits[32];          // per row of a block: columns reached, kept, passed, handing on
  unsigned row_risk[32];       // ... kept from below at a value that may lie past the edge's end
  int2 base[2][32];            // per row: first right edge's and first top edge's value
  double bot[2][32];           // values rows enter / leave the block with
  int up_j[2][kWalkCap];       // live chunks of the row below / of the row being made
  double up_v[2][kWalkCap][32];
  double stage[2][kWalkStage];
  double2 vals[2][kWalkVals];
  unsigned short list[kWalkVals];
  double dead_row[32], spare_row[32];
  int nup, lost, scan_lo, scan_hi;  // scan of a piece's first row: chunks found, among which
};
constexpr size_t kWalkSmem = (sizeof(WalkShared) + 127) / 128 * 128;

__device__ __forceinline__ void walk_helper_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(32 * kWalkHelpers) : "memory");
}

// ------------------------------------------------------------------ helpers (warps 1..7)

// Skip threshold of the edges of a segment with squared length A: an edge whose far end point
// lies farther than this (squared) from the other curve's point is certainly dead.  The point
// is then more than rad + 0.004 (rad + length) from every point of the segment, a relative
// margin of 1e-6 of the squared distances involved, while the FP64 code that computes the
// edge errs by about 1e-8 of them (a discriminant at 0) and never calls such an edge live.
// No skipping for degenerate segments (their free interval is [0, 1] at any radius), near the
// ends of the exponent range, or where distances are lost in the coordinates' rounding.
// (Lengths in FP32, rounded up, where they fit: an FP64 root is a third of the stage's time.)
__device__ __forceinline__ double walk_threshold(double rad, double A, double mag) {
  const double len = A > 1e-30 && A < 1e30 ? 1.0005 * (double)sqrtf((float)A) : __dsqrt_rn(A);
  const double s = rad + len;
  const double t = fmax(1.01 * s * s, 1e-14 * mag * mag);
  return A > 1e-200 && t < 1e200 ? t : (double)INFINITY;
}

__device__ __forceinline__ void walk_prefetch(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Tile of block (bi, bj), all helpers; tid in [0, 32 H).
template <int D, int KIND>
__device__ __forceinline__ void walk_tile(const PairDesc& pd, WalkShared* sh, int slot, int bi,
                                          int bj, int tid) {
  const int lane = tid & 31, hw = tid >> 5;
  constexpr int NT = 32 * kWalkHelpers;
  constexpr bool dfd = KIND == K_DFD;
  double* P = sh->stage[slot];
  double* Q = P + kWalkPts;
  double* ra = Q + kWalkPts;  // row segments: A, 0.5/A, threshold
  double* rinv = ra + 32;
  double* rthr = rinv + 32;
  double* ca = rthr + 32;     // column segments
  double* cinv = ca + 32;
  double* cthr = cinv + 32;
  const int R = dfd ? pd.n1 : pd.n1 - 1, C = dfd ? pd.n2 : pd.n2 - 1;
  const int i0 = bi << 5, j0 = bj << 5;
  const int nr = min(32, R - i0), nc = min(32, C - j0);
  {
    // points 32 bi .. 32 bi + 32 (clamped to the curve's end; clamped ones feed no cell)
    static_assert(33 * 3 <= NT, "one point coordinate a thread");
    const long long pe = (long long)pd.n1 * D - 1, qe = (long long)pd.n2 * D - 1;
    if (tid < 33 * D) {
      P[tid] = __ldg(pd.P + min((long long)i0 * D + tid, pe));
      Q[tid] = __ldg(pd.Q + min((long long)j0 * D + tid, qe));
    }
    // the points of the blocks right and up, which come next (16 doubles a line)
    if (tid >= 192 && tid < 192 + 16) {
      const int e = (tid - 192) * 16;
      walk_prefetch(pd.P + min((long long)(i0 + 32) * D + e, pe));
      walk_prefetch(pd.Q + min((long long)(j0 + 32) * D + e, qe));
    }
  }
  if (hw == 3) {
    sh->mask[slot][lane] = make_uint4(0u, 0u, 0u, 0u);
    if (KIND == K_DEC) sh->risk[slot][lane] = make_uint4(0u, 0u, 0u, 0u);
    if (lane == 0) sh->cnt[slot] = 0;
  }
  if (!dfd && (hw == 4 || hw == 5)) {
    // segment constants from prep_kernel's records
    const bool col = hw == 5;
    const int e = min((col ? j0 : i0) + lane, (col ? C : R) - 1);
    const double2 rec = __ldg(col ? sh->seg_c + (size_t)e * sh->step_c : sh->seg_r + (size_t)e * sh->step_r);
    const double* x = (col ? pd.Q : pd.P) + (size_t)(e + 1) * D;
    double mag = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) mag = fmax(mag, fabs(__ldg(x + k)));
    double* a = col ? ca : ra;
    a[lane] = rec.x;
    a[32 + lane] = rec.y;
    a[64 + lane] = walk_threshold(sh->rad, rec.x, mag);
  }
  walk_helper_sync();

  if constexpr (dfd) {
    // point distances are cheap: every cell
    double* W = reinterpret_cast<double*>(sh->vals[slot]);
    const double U = sh->level;
    for (int r = hw; r < nr; r += kWalkHelpers) {
      const double w = dist_sq<D>(P + r * D, Q + lane * D);
      W[r * 32 + lane] = w;
      const unsigned m = __ballot_sync(kFull, (lane < nc) & (w <= U));
      if (lane == 0) sh->mask[slot][r].w = m;
    }
  } else {
    // which edges can be live: lane = column; the warp's rows hw + 7 m together (independent
    // tests), then one allocation for all
    constexpr int M = (32 + kWalkHelpers - 1) / kWalkHelpers;
    unsigned br[M], bt[M];
    int n = 0;
    {
      double q[D];
#pragma unroll
      for (int k = 0; k < D; ++k) q[k] = Q[(lane + 1) * D + k];
      const double ct = cthr[lane];
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int r = min(hw + m * kWalkHelpers, 31);
        const bool in = (lane < nc) & (hw + m * kWalkHelpers < nr);
        const double s = dist_sq<D>(P + (r + 1) * D, q);
        br[m] = __ballot_sync(kFull, in & !(s > ct));
        bt[m] = __ballot_sync(kFull, in & !(s > rthr[r]));
        n += __popc(br[m]) + __popc(bt[m]);
      }
    }
    if (n) {
      const unsigned lt = (1u << lane) - 1u;
      int at = 0;
      if (lane == 0) at = atomicAdd(&sh->cnt[slot], n);
      at = bcast(at);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int r = hw + m * kWalkHelpers;
        const int kr = __popc(br[m]), kt = __popc(bt[m]);
        if (br[m] >> lane & 1u) sh->list[at + __popc(br[m] & lt)] = (unsigned short)(r << 5 | lane);
        if (bt[m] >> lane & 1u)
          sh->list[at + kr + __popc(bt[m] & lt)] = (unsigned short)(1024 | r << 5 | lane);
        if ((lane == 0) & (kr + kt > 0)) {
          sh->mask[slot][r] = make_uint4(br[m], bt[m], 0u, 0u);
          sh->base[slot][r] = make_int2(at, at + kr);
        }
        at += kr + kt;
      }
    }
    walk_helper_sync();

    const int cnt = sh->cnt[slot];
    const double level = sh->level;
    const bool mat = KIND == K_DEC && sh->mat != 0, filt = KIND == K_DEC && sh->filter != 0;
    unsigned cells64 = 0;
    if (*(volatile int*)&sh->cancel[slot]) return;
    for (int k = tid; k < cnt; k += NT) {
      const int e = sh->list[k], r = (e >> 5) & 31, c = e & 31;
      const bool top = e >= 1024;
      // right edge: p_{i+1} against q_j q_{j+1}; top edge: q_{j+1} against p_i p_{i+1}
      const double* x = top ? Q + (c + 1) * D : P + (r + 1) * D;
      const double* a = top ? P + r * D : Q + c * D;
      double di[D];
#pragma unroll
      for (int d = 0; d < D; ++d) di[d] = __dsub_rn(a[D + d], a[d]);
      const double* seg = top ? ra + r : ca + c;
      bool live;
      if constexpr (KIND == K_DEC) {
        double lo, hi;
        // the FP32 filter's certain answers need no FP64 (rfd_filter.h)
        const int cls = filt ? interval_class32<D>(x, a, di, seg[0], level) : 0;
        if (cls == 0) {
          free_interval<D>(x, a, di, seg[0], seg[32], level, lo, hi, mat);
          cells64 += filt;
        } else {
          lo = cls == 1 ? -1.0 : 0.0;
          hi = cls == 1 ? -2.0 : 1.0;
        }
        sh->vals[slot][k] = make_double2(lo, hi);
        live = !(lo < 0.0);
        uint4* risk = &sh->risk[slot][r];
        if (live & (hi < 1.0)) atomicOr(top ? &risk->z : &risk->x, 1u << c);
        if (live & !top & (lo > 0.0)) atomicOr(&risk->y, 1u << c);
      } else {
        const double w = pt_seg_sq<D>(x, a, di, seg[0]);
        reinterpret_cast<double*>(sh->vals[slot])[k] = w;
        live = w <= level;
      }
      if (live) atomicOr(top ? &sh->mask[slot][r].w : &sh->mask[slot][r].z, 1u << c);
    }
    // (edges; halved by the reader: at most the cells listed)
    if (cells64) atomicAdd(&sh->cells64, (unsigned long long)cells64);
  }
}

// Bounds of a curve's chunks (points 32 J - 1 .. 32 J + 32), one warp a chunk; a chunk with a
// degenerate segment, whose free interval is [0, 1] at any radius, is unbounded.
template <int D>
__device__ void walk_ball(const double* X, int n, int j, WalkBall* out) {
  const int lane = threadIdx.x & 31;
  double lo[D], hi[D];
#pragma unroll
  for (int k = 0; k < D; ++k) {
    lo[k] = (double)INFINITY;
    hi[k] = -(double)INFINITY;
  }
  bool odd = false;
  for (int q = (j << 5) - 1 + lane; q <= (j << 5) + 32; q += 32) {
    if (q < 0 || q >= n) continue;
    double A = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const double v = X[(size_t)q * D + k];
      lo[k] = fmin(lo[k], v);
      hi[k] = fmax(hi[k], v);
      odd |= !(fabs(v) < 1e140);
      if (q + 1 < n) {
        const double d = X[(size_t)(q + 1) * D + k] - v;
        A += d * d;
      }
    }
    if (q + 1 < n) odd |= !(A > 1e-200);
  }
  double rad = 0.0, x[D];
#pragma unroll
  for (int k = 0; k < D; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] = fmin(lo[k], __shfl_xor_sync(kFull, lo[k], o));
      hi[k] = fmax(hi[k], __shfl_xor_sync(kFull, hi[k], o));
    }
    x[k] = 0.5 * (lo[k] + hi[k]);
    rad += 0.25 * (hi[k] - lo[k]) * (hi[k] - lo[k]);
  }
  odd = __any_sync(kFull, odd);
  if (lane == 0) {
    WalkBall b;
    b.x[2] = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) b.x[k] = x[k];
    b.rad = odd ? (double)INFINITY : 1.000001 * sqrt(rad);
    *out = b;
  }
}

// The row below block row bi, as far as it can be live (see the head comment): chunks into list
// `to`, in no order (the propagator sorts them); sh->nup of them, sh->lost if some did not fit.
template <int D>
__device__ void walk_scan(const PairDesc& pd, WalkShared* sh, int to, int bi, int tid) {
  const int lane = tid & 31, hw = tid >> 5;
  const int kind = sh->kind;
  const bool dfd = kind == K_DFD;
  const int C = dfd ? pd.n2 : pd.n2 - 1, nbc = (C + 31) >> 5;
  const double level = sh->level;
  if (tid == 0) sh->nup = sh->lost = 0;
  walk_helper_sync();
  // segment kinds: point 32 bi against the columns' segments; DFD: point 32 bi - 1
  const double* xp = pd.P + (size_t)((bi << 5) - (dfd ? 1 : 0)) * D;
  double x[D];
  double mag = 0.0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    x[k] = __ldg(xp + k);
    mag = fmax(mag, fabs(x[k]));
  }
  const double dead = kind == K_DEC ? kDecDead : kFltMax;
  const int j1 = min(nbc, sh->scan_hi + 1);
  for (int jb = max(0, sh->scan_lo) + 32 * hw; jb < j1; jb += 32 * kWalkHelpers) {
   // 32 chunks' bounds at once, then the chunks in reach one by one
   bool reach = false;
   if (jb + lane < j1) {
    const WalkBall* b = pd.balls + jb + lane;
    double t[D];
#pragma unroll
    for (int k = 0; k < D; ++k) t[k] = x[k] - __ldg(&b->x[k]);
    const double far = 1.00001 * (sh->rad + __ldg(&b->rad)) + 1e-7 * mag;
    reach = !(sq_sum<D>(t) > far * far);
   }
   unsigned todo = __ballot_sync(kFull, reach);
   while (todo) {
    const int j = jb + __ffs(todo) - 1, c = (j << 5) + lane;
    todo &= todo - 1;
    double v = dead;
    if (c < C) {
      if (dfd) {
        auto weight = [&](int q) {
          double b[D];
#pragma unroll
          for (int e = 0; e < D; ++e) b[e] = __ldg(pd.Q + (size_t)q * D + e);
          return dist_sq<D>(x, b);
        };
        const double w = weight(c), l = weight(max(c - 1, 0));
        v = l < w ? l : w;
        v = v <= level ? v : dead;
      } else {
        double a[D], di[D];
#pragma unroll
        for (int e = 0; e < D; ++e) {
          a[e] = __ldg(pd.Q + (size_t)c * D + e);
          di[e] = __dsub_rn(__ldg(pd.Q + (size_t)(c + 1) * D + e), a[e]);
        }
        const double A = sq_sum<D>(di);
        if (kind == K_DEC) {
          double lo, hi;
          free_interval<D>(x, a, di, A, __ddiv_rn(0.5, A), level, lo, hi, sh->mat != 0);
          v = lo < 0.0 ? dead : lo;
        } else {
          const double w = pt_seg_sq<D>(x, a, di, A);
          v = w <= level ? w : dead;
        }
      }
    }
    if (sh->flat && v < dead) v = 0.0;
    if (!__any_sync(kFull, v < (kind == K_DEC ? kDecLive : kFltMax))) continue;
    int at = 0;
    if (lane == 0) at = atomicAdd(&sh->nup, 1);
    at = bcast(at);
    if (at < kWalkCap) {
      sh->up_v[to][at][lane] = v;
      if (lane == 0) sh->up_j[to][at] = j;
    } else if (lane == 0) {
      sh->lost = 1;
    }
   }
  }
}

// Helper warps: tiles as requested, until kStop.
__device__ void walk_helpers(const WaveArgs& wa, WalkShared* sh) {
  const int tid = threadIdx.x - 32, lane = tid & 31;
  unsigned seq = 0;
  for (;;) {
    const int slot = seq & 1;
    if (!mbar_wait(&sh->req[slot], (seq >> 1) & 1, wa, clock64())) break;
    const int bi = *(volatile int*)&sh->req_i[slot], bj = *(volatile int*)&sh->req_j[slot];
    if (bi == kStop) break;
    const PairDesc pd = sh->pd;
    if (bi == kScan) {
      if (pd.d == 2) walk_scan<2>(pd, sh, sh->scan_to, bj, tid);
      else walk_scan<3>(pd, sh, sh->scan_to, bj, tid);
    } else if (sh->kind == K_DEC) {
      if (pd.d == 2) walk_tile<2, K_DEC>(pd, sh, slot, bi, bj, tid);
      else walk_tile<3, K_DEC>(pd, sh, slot, bi, bj, tid);
    } else if (sh->kind == K_VEFD) {
      if (pd.d == 2) walk_tile<2, K_VEFD>(pd, sh, slot, bi, bj, tid);
      else walk_tile<3, K_VEFD>(pd, sh, slot, bi, bj, tid);
    } else {
      if (pd.d == 2) walk_tile<2, K_DFD>(pd, sh, slot, bi, bj, tid);
      else walk_tile<3, K_DFD>(pd, sh, slot, bi, bj, tid);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh->full[slot]);
    ++seq;
  }
}

// ------------------------------------------------------------------ propagator (warp 0)

template <int KIND>
__device__ __forceinline__ double walk_dead() {
  return KIND == K_DEC ? kDecDead : kFltMax;
}
// Live values are below the dead one by construction (masked edges only); for the decision the
// high word decides.
template <int KIND>
__device__ __forceinline__ bool walk_live(double v) {
  return KIND == K_DEC ? __double2hiint(v) < __double2hiint(kDecLive) : v < kFltMax;
}
// a < b for values >= 0 (or -0, which sorts first) as integers: shorter than an FP64 compare.
__device__ __forceinline__ bool walk_less(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}

__device__ __forceinline__ double walk_min(double a, double b) { return walk_less(a, b) ? a : b; }
__device__ __forceinline__ double walk_max(double a, double b) { return walk_less(a, b) ? b : a; }

// Place of a listed edge's value: the row's first one and the listed edges left of column c.  (A
// column without a listed edge, or a row that lists none and whose place is stale, gives some
// place within the tile; its value is not used.)
__device__ __forceinline__ unsigned walk_place(int first, unsigned listed, int c) {
  return min((unsigned)first + __popc(listed & ((1u << c) - 1u)), (unsigned)kWalkVals - 1u);
}

// Row r of a block's decision, every value formed (lane = column).  F: value handed up by the row
// below, replaced by this row's; V: its live columns.  in: whether the row enters the block
// live, with value x0.  y: value this lane's column hands to the right; Y: the columns that
// hand on a live one.  The value runs right through top edges: column j hands on t.lo when it
// is live from below, else max(t.lo, x) if the incoming x is at most t.hi; repeated until no
// column changes (as often as the longest run of columns without support from below).
__device__ __forceinline__ void walk_row(const WalkShared* sh, int slot, int r, bool in, double x0,
                                         double& F, unsigned& V, double& y, unsigned& Y) {
  const int lane = threadIdx.x & 31;
  const unsigned bit = 1u << lane;
  const uint4 m = sh->mask[slot][r];
  const int2 base = sh->base[slot][r];
  const double2 er = sh->vals[slot][walk_place(base.x, m.x, lane)];
  const double2 et = sh->vals[slot][walk_place(base.y, m.y, lane)];
  const bool br = (m.z & bit) != 0u, bt = (m.w & bit) != 0u, up = (V & bit) != 0u;
  const double first = in ? x0 : kDecDead;  // what enters column 0
  double x;
  y = bt & up ? et.x : kDecDead;
  for (;;) {
    x = __shfl_up_sync(kFull, y, 1);
    x = lane == 0 ? first : x;
    const bool ends = !bt | (!up & walk_less(et.y, x));
    const bool own = up | !walk_less(et.x, x);
    double yn = own ? et.x : x;
    yn = ends ? kDecDead : yn;
    const bool moved = walk_less(yn, y) | walk_less(y, yn);
    y = yn;
    if (!__any_sync(kFull, moved)) break;
  }
  const bool xl = walk_live<K_DEC>(x);
  const bool ok = br & (xl | !walk_less(er.y, F));
  const bool own = xl | !walk_less(er.x, F);
  const double f = own ? er.x : F;
  F = ok ? f : kDecDead;
  V = __ballot_sync(kFull, ok);
  Y = __ballot_sync(kFull, walk_live<K_DEC>(y));
}

// Rows r .. nr - 1 of a block as far as bits settle them (decision and flat sweeps).  First the
// live columns, row by row, as if no value stood in the way of another: whether a value arrives
// at a column is a carry chain (generate: live from below and the top edge free; propagate: top
// edge free), one addition for the row's 32 columns.  A value can stand in the way only where
// an edge that ends before 1 is kept from below by a value above 0, or passed without support
// from below; bits say where that may be (few places in a thin band), and there the values are
// formed and compared, lane = row.  The values handed on are formed last, a column of the last
// row from its run of rows.
// Returns nr, or the first row where a value does meet an edge that ends before it: what is handed
// on is then as of the row before.
template <int KIND>
__device__ __forceinline__ int walk_bits(WalkShared* sh, int slot, int r, int nr, unsigned bmask,
                                         const double* bin, double* bout, double& F, unsigned& V,
                                         unsigned& omask, unsigned& Y) {
  const int lane = threadIdx.x & 31;
  const unsigned bit = 1u << lane;
  const double dead = walk_dead<KIND>();
  // from the first row that has something live to the last (a loop of few instructions: code that
  // runs once a block is fetched at 5 cycles an instruction)
  const unsigned entries = bmask & (0xffffffffu << r);
  const int r0 = V ? r : __ffs(entries) - 1;
  int r1 = r0;
  unsigned v = V, yl = 0u;
  {
    unsigned above = KIND == K_DEC ? __ballot_sync(kFull, walk_live<KIND>(F) & (F > 0.0)) : 0u;
    unsigned in = entries >> r0;
    uint2 m = *reinterpret_cast<const uint2*>(&sh->mask[slot][r0].z), k = make_uint2(0u, 0u);
    if (KIND == K_DEC) k = *reinterpret_cast<const uint2*>(&sh->risk[slot][r0].x);
#pragma unroll 2
    do {
      const int rn = min(r1 + 1, 31);
      const uint2 mn = *reinterpret_cast<const uint2*>(&sh->mask[slot][rn].z);
      uint2 kn = k;
      if (KIND == K_DEC) kn = *reinterpret_cast<const uint2*>(&sh->risk[slot][rn].x);
      const unsigned gen = v & m.y;
      const unsigned X = (m.y + gen + (in & 1u)) ^ m.y ^ gen;  // live values arriving
      const unsigned any = X | v;
      yl = m.y & any;
      const unsigned ok = KIND == K_DFD ? (yl | X) : m.x & any;
      sh->row_bits[r1] = make_uint4(X, ok, X & ~v & m.y, yl);
      if (KIND == K_DEC) {
        const unsigned held = above & ~X;  // columns kept from below, at values that may exceed 0
        sh->row_risk[r1] = ok & held & k.x;
        above = ok & (k.y | held);
      }
      v = ok;
      m = mn;
      k = kn;
      in >>= 1;
      ++r1;
    } while ((r1 < nr) & ((v | in) != 0u));
  }
  __syncwarp();
  const bool mine = (lane >= r0) & (lane < r1);
  uint4 rb = sh->row_bits[lane];
  if (!mine) rb = make_uint4(0u, 0u, 0u, 0u);
  unsigned top = r1 == nr ? v : 0u;
  unsigned out = __ballot_sync(kFull, (rb.w >> 31) != 0u);
  if (KIND != K_DEC) {
    if (rb.w >> 31) bout[lane] = 0.0;
    F = top & bit ? 0.0 : dead;
  } else {
    const uint4 m = sh->mask[slot][lane];
    const int2 base = sh->base[slot][lane];
    const double2* vals = sh->vals[slot];
    bool clash = false;
    // passes, left to right, in the rows where one meets an edge that ends before 1 or is the
    // last column's
    unsigned todo = rb.z & (sh->risk[slot][lane].z | 0x80000000u) ? rb.z : 0u;
    double x = 0.0;
    int before = -2;  // column passed last, x what it handed on
    unsigned rows = __ballot_sync(kFull, todo != 0u);
    if ((int)__reduce_max_sync(kFull, __popc(todo)) > 1 + __popc(rows)) {
      // few rows with long passes: these one by one, lane = column, the largest start of a pass so
      // far by a scan over the columns (about what two steps of the loop below take)
      for (; rows; rows &= rows - 1u) {
        const int q = __ffs(rows) - 1;
        const uint4 b = sh->row_bits[q], mq = sh->mask[slot][q];
        const double2 t = vals[walk_place(sh->base[slot][q].y, mq.y, lane)];
        const bool pass = (b.z & bit) != 0u;
        double g = (lane == 0) & pass ? walk_max(t.x, bin[q]) : t.x;
        const unsigned heads = ~b.z | 1u;
        const int run = lane - (31 - __clz(heads & (bit | (bit - 1u))));
#pragma unroll 1
        for (int d = 1; d < 32; d <<= 1) {
          const double h = __shfl_up_sync(kFull, g, d);
          g = run >= d ? walk_max(g, h) : g;
        }
        double from = __shfl_up_sync(kFull, g, 1);
        from = lane == 0 ? bin[q] : from;
        const bool hits = __any_sync(kFull, pass & walk_less(t.y, from));
        const double end = __shfl_sync(kFull, g, 31);
        clash |= (lane == q) & hits;
        x = lane == q ? end : x;
        before = (lane == q) & (int)(b.z >> 31) ? 31 : before;
      }
      todo = 0u;
    }
    while (__any_sync(kFull, todo != 0u)) {
      const int c = todo ? __ffs(todo) - 1 : 0;
      const double own = c == 0 ? bin[lane] : vals[walk_place(base.y, m.y, c - 1)].x;
      const double2 t = vals[walk_place(base.y, m.y, c)];
      const double from = before == c - 1 ? x : own;
      clash |= (todo != 0u) & walk_less(t.y, from);
      x = todo ? walk_max(t.x, from) : x;
      before = todo ? c : before;
      todo &= todo - 1u;
    }
    if (rb.w >> 31) bout[lane] = before == 31 ? x : vals[walk_place(base.y, m.y, 31)].x;
    // values kept from below that may lie past the edge's end: down the column to where the run
    // started, the largest start on the way
    todo = mine ? sh->row_risk[lane] : 0u;
    int row = lane;  // row looked at last, of the run under cell (lane, lowest bit of todo)
    double f = 0.0;
    unsigned cols = __reduce_or_sync(kFull, todo);
    if (cols && __popc(cols) <= 2) {
      // one or two columns: each by a scan over its rows
      for (; cols; cols &= cols - 1u) {
        const int c = __ffs(cols) - 1;
        const double2 e = vals[walk_place(base.x, m.x, c)];
        const bool reached = (rb.x >> c & 1u) != 0u;
        const double f0 = __shfl_sync(kFull, F, c);
        const bool below = (lane == r0) & !reached;
        double g = below ? walk_max(e.x, f0) : e.x;
        const unsigned heads = __ballot_sync(kFull, reached | (lane <= r0) | !(rb.y >> c & 1u));
        const int run = lane - (31 - __clz(heads & (bit | (bit - 1u))));
#pragma unroll 1
        for (int d = 1; d < 32; d <<= 1) {
          const double h = __shfl_up_sync(kFull, g, d);
          g = run >= d ? walk_max(g, h) : g;
        }
        double under = __shfl_up_sync(kFull, g, 1);
        under = below ? f0 : under;
        clash |= ((todo >> c & 1u) != 0u) & walk_less(e.y, under);
      }
      todo = 0u;
    }
    while (__any_sync(kFull, todo != 0u)) {
      const int c = todo ? __ffs(todo) - 1 : 0;
      const double f0 = __shfl_sync(kFull, F, c);
      row = max(row - 1, r0 - 1);
      const int q = max(row, r0);
      const double lo = vals[walk_place(sh->base[slot][q].x, sh->mask[slot][q].x, c)].x;
      f = walk_max(f, row < r0 ? f0 : lo);
      const bool start = (row < r0) | ((sh->row_bits[q].x >> c & 1u) != 0u);
      const double hi = vals[walk_place(base.x, m.x, c)].y;
      clash |= (todo != 0u) & start & walk_less(hi, f);
      todo = start ? todo & (todo - 1u) : todo;
      row = start ? lane : row;
      f = start ? 0.0 : f;
    }
    const unsigned bad = __ballot_sync(kFull, clash);
    if (bad) {
      // up to there
      nr = __ffs(bad) - 1;
      if (nr == r0) return nr;
      r1 = nr;
      const uint4 b = sh->row_bits[nr - 1];
      top = b.y;
      yl = b.w;
      out &= (1u << nr) - 1u;
    }
    // the last row's values
    double Fn = dead;
    for (unsigned cols = top; cols; cols &= cols - 1u) {
      const int c = __ffs(cols) - 1;
      const bool reached = (rb.x >> c & 1u) != 0u;
      const bool below = (lane == r0) & !reached;  // the run starts in the row below
      const double lo = vals[walk_place(base.x, m.x, c)].x, f0 = __shfl_sync(kFull, F, c);
      const unsigned heads = __ballot_sync(kFull, reached | (lane == r0) | !(rb.y >> c & 1u));
      const int head = 31 - __clz(heads & (nr == 32 ? kFull : (1u << nr) - 1u));
      // (rows head .. nr - 1 are the run; others take no part)
      double g = (lane >= head) & (lane < nr) ? lo : 0.0;
      g = (lane == head) & below ? walk_max(g, f0) : g;
#pragma unroll 1
      for (int d = 16; d > 0; d >>= 1) g = walk_max(g, __shfl_xor_sync(kFull, g, d));
      Fn = lane == c ? g : Fn;
    }
    F = Fn;
  }
  V = top;
  omask |= out;
  Y = r1 == nr ? yl : 0u;
  __syncwarp();
  return nr;
}

// A block of a min-max sweep with its values: a skewed sweep (lane = row, step t: column t -
// lane) over the anti-diagonals that have a live value.  upv / V: the row below (values, live
// columns); rows enter with bin where bmask says so and leave with bout; out: the row handed on.
// y, f: last column's and row's values of this lane's row.
template <int KIND>
__device__ __forceinline__ void walk_values(const WalkShared* sh, int slot, int nr, int nc,
                                            const double* upv, unsigned V, unsigned bmask,
                                            const double* bin, double* bout, unsigned& omask,
                                            double* out, double& y, double& f) {
  const int lane = threadIdx.x & 31;
  const double dead = kFltMax;
  const double* vals = reinterpret_cast<const double*>(sh->vals[slot]);
  const uint4 m = sh->mask[slot][lane];
  int kr = 0, kt = lane * 32;
  if (KIND == K_VEFD) {
    const int2 base = sh->base[slot][lane];
    kr = max(min(base.x, kWalkVals), 0);  // (stale where the row lists nothing)
    kt = max(min(base.y, kWalkVals), 0);
  }
  double bot = bmask >> lane & 1u ? bin[lane] : dead, carry = dead;
  out[lane] = dead;
  __syncwarp();
  const bool store = lane == nr - 1;
  int t = min(V ? __ffs(V) - 1 : 64, bmask ? __ffs(bmask) - 1 : 64);
  // (columns skipped at the start: their listed edges too)
  auto skip = [&](int c) {
    if (KIND == K_VEFD && c > 0) {
      const unsigned below = c > 31 ? kFull : (1u << c) - 1u;
      kr += __popc(m.x & below);
      kt += __popc(m.y & below);
    }
  };
  skip(t - lane);
  while (t < nr + nc - 1) {
#pragma unroll 2
    for (int u = 0; u < 4; ++u, ++t) {
      const int c = t - lane;
      const bool act = (unsigned)c < (unsigned)nc;
      const unsigned bit = act ? 1u << c : 0u;
      double left = __shfl_up_sync(kFull, carry, 1);
      const double low = upv[t & 31];
      left = lane == 0 ? low : left;
      const double in = walk_min(left, bot);
      double ncarry, nbot;
      if (KIND == K_VEFD) {
        const double wr = vals[kr], wt = vals[kt];
        kr += (m.x & bit) != 0u;
        kt += (m.y & bit) != 0u;
        ncarry = walk_max(wr, in);
        ncarry = (m.z & bit) != 0u ? ncarry : dead;
        nbot = walk_max(wt, in);
        nbot = (m.w & bit) != 0u ? nbot : dead;
      } else {
        const double w = vals[kt + max(min(c, 31), 0)];
        nbot = walk_max(w, in);
        nbot = (m.w & bit) != 0u ? nbot : dead;
        ncarry = walk_min(nbot, bot);
      }
      carry = act ? ncarry : carry;
      bot = act ? nbot : bot;
      if (act & store) out[c] = carry;
    }
    // rows at work in step t, or handing a live value to one that is
    const bool busy = ((lane <= t) & (lane + 31 >= t) & (bot < dead)) |
                      ((lane < t) & (lane + 32 >= t) & (lane < 31) & (carry < dead));
    if (!__any_sync(kFull, busy)) {
      // all dead: on to the next live input, if any
      const unsigned fb = __ballot_sync(kFull, (lane > t) & (bot < dead));
      const unsigned fu = t < 32 ? V & (0xffffffffu << t) : 0u;
      if (!(fb | fu)) break;
      const int to = __ffs(fb | fu) - 1;
      if (KIND == K_VEFD) {
        // listed edges of the columns jumped over
        const int c0 = min(max(t - lane, 0), 32), c1 = min(max(to - lane, 0), 32);
        const unsigned b1 = c1 > 31 ? kFull : (1u << c1) - 1u, b0 = c0 > 31 ? kFull : (1u << c0) - 1u;
        kr += __popc(m.x & b1 & ~b0);
        kt += __popc(m.y & b1 & ~b0);
      }
      t = to;
    }
  }
  __syncwarp();
  omask = __ballot_sync(kFull, (bot < dead) & (lane < nr));
  if (lane < nr) bout[lane] = bot;
  // (a sweep that ended before lane 31 came to the last column, all dead from there on, leaves it
  // what it handed up from an earlier column; the other lanes' live values keep the sweep going)
  y = bot;
  f = t - lane >= nc ? carry : dead;
  __syncwarp();
}

// Walk of one CTA: requests outstanding, and the list of the row below.
struct Walk {
  unsigned seq_p, seq_c;  // tiles requested, taken
  int pi, pj;             // the outstanding request (pi < 0: none)
  int cur, n;             // list of the row below: buffer and live chunks
  long long t0;           // cycle the running walk began
  int blocks, effort;     // its blocks, and with their listed edges (256 count as a block)
  int rec_from, rec_end;  // block rows whose records this sweep can be met at
  // where an earlier sweep's band ran: this member's piece, cut so that pieces take equal
  // stretches of the band, and the chunks it entered it in (lo > hi: not known)
  WalkCut cut;
  int near_lo, near_hi;
  // of the phase (walk_pair): its rule of giving up, cycle past which it is given up, cycles that the
  // strips would need, cycles that a piece may take for a block ahead (0: any); whether the
  // deadline has passed (the same for all members)
  int rule;
  long long deadline;
  float strips, pace;
  bool late;
  // the group's sweeps so far, and its word that holds the number of the last one whose end was
  // known before every piece had been walked
  unsigned sweeps;
  unsigned* stop;
};

enum WalkStatus : int { WALK_OK = 0, WALK_ERROR, WALK_GIVE_UP, WALK_MET, WALK_UNSETTLED, WALK_STOPPED };
// How a piece is walked: alone (the whole grid); the first time from what could be live, or
// from the true start, recording every block row's list; again, until it meets a record.
enum WalkMode : int { WALK_ALONE = 0, WALK_RECORD = 1, WALK_AGAIN = 2 };

// Rules of giving up (walk_slow), by what the strips would cost instead:
//   WALK_BY_EFFORT  blocks and listed edges against the blocks the walk has come ahead: a thin band
//                   lists a few hundred edges a block and goes from block to block right or up (a
//                   pair of many, each walked by one CTA: the strips' time is the call's then);
//   WALK_BY_REST    a lone CTA's walk, once a twelfth of the strips' time has passed (60 us at
//                   most): if the rest takes longer than the strips (what is spent is spent; 1.15:
//                   rates vary along a band).  The rest is the blocks still ahead at the rate so
//                   far, or the rows still to come with as many chunks as the list has now;
//   WALK_BY_TIME    a group's: the phase's deadline; and a piece, where `pace` says so, against a thin
//                   band's rate, which is about 5 us a block row or column for the decision and 8
//                   for the others.  A wide band's blocks cost 4 to 16 us each (most of their edges
//                   listed), a row of them tells (150 x 140 unrelated points, decide_noalloc: 205
//                   us walked, 100 on the strips, 130 given up).
enum WalkRule : int { WALK_BY_EFFORT = 0, WALK_BY_REST, WALK_BY_TIME };
// ahead, total: blocks come ahead, of the grid's rows and columns; chunks: of the list; rows, left: the
// piece's, and those still to come.  Asked every fourth block (the code that runs once a block is
// fetched anew: asked every block it took 7 % of a decision).
__device__ __forceinline__ bool walk_slow(const Walk& w, int ahead, int total, int chunks, int rows,
                                          int left) {
  if (w.rule == WALK_BY_EFFORT) return w.effort > 64 + 4LL * (ahead - 1);
  constexpr float us = kWalkClock;
  const long long now = clock64();
  const float spent = (float)(now - w.t0), blocks = (float)w.blocks;
  const float to_come = spent * (float)(chunks * left);  // (times the blocks)
  if (w.rule == WALK_BY_REST)
    return spent > fminf(w.strips / 12.f, 60.f * us) &&
           (spent * (float)(total - ahead) > 1.15f * w.strips * (float)ahead ||
            to_come > 1.15f * w.strips * blocks);
  if (now > w.deadline) return true;
  if (!(w.pace > 0.f)) return false;
  const float may = fmaxf(15.f * us + w.pace * (float)ahead, 0.12f * w.strips);
  const float may_all = fmaxf(15.f * us + w.pace * (float)(2 * rows), 0.12f * w.strips);
  return spent > may || (spent > 10.f * us && to_come > (1.5f * may_all - spent) * blocks);
}
// Tells the other members that this sweep's end is known, or that it is given up.
__device__ __forceinline__ void walk_stop(const Walk& w) {
  if ((threadIdx.x & 31) == 0) *(volatile unsigned*)w.stop = w.sweeps;
  __syncwarp();
}

__device__ __forceinline__ void walk_request(WalkShared* sh, Walk& w, int i, int j) {
  if ((threadIdx.x & 31) == 0) {
    const int slot = w.seq_p & 1;
    *(volatile int*)&sh->req_i[slot] = i;
    *(volatile int*)&sh->req_j[slot] = j;
    *(volatile int*)&sh->cancel[slot] = 0;
    mbar_arrive(&sh->req[slot]);
  }
  __syncwarp();
  ++w.seq_p;
  w.pi = i;
  w.pj = j;
}
// The propagator's wait for a tile (bounded).  It polls: the helpers' waits suspend
// (mbarrier.try_wait), but this one is on the sweep's chain.
__device__ __forceinline__ bool walk_wait(unsigned long long* b, unsigned parity, const WaveArgs& wa) {
  const long long t0 = clock64();
  for (int it = 0;; ++it) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(b)), "r"(parity)
        : "memory");
    if (ok) return true;
    int bad = 0;
    if ((threadIdx.x & 31) == 0)
      bad = clock64() - t0 > wa.spin_cycles || ((it & 255) == 255 && ld_volatile(wa.error));
    if (__shfl_sync(kFull, bad, 0)) {
      if ((threadIdx.x & 31) == 0) atomicExch(wa.error, 1);
      return false;
    }
  }
}
// Waits for the outstanding tile; its slot, or -1 on an error.
__device__ __forceinline__ int walk_take(const WaveArgs& wa, WalkShared* sh, Walk& w) {
  const int slot = w.seq_c & 1;
  if (!walk_wait(&sh->full[slot], (w.seq_c >> 1) & 1, wa)) return -1;
  ++w.seq_c;
  w.pi = -1;
  return slot;
}
__device__ __forceinline__ bool walk_drop(const WaveArgs& wa, WalkShared* sh, Walk& w) {
  if (w.pi < 0) return true;
  if ((threadIdx.x & 31) == 0) *(volatile int*)&sh->cancel[w.seq_c & 1] = 1;
  __syncwarp();
  return walk_take(wa, sh, w) >= 0;
}
// The tile of block (i, j): taken if it is the outstanding request.
__device__ __forceinline__ int walk_get(const WaveArgs& wa, WalkShared* sh, Walk& w, int i, int j) {
  if ((w.pi != i) | (w.pj != j)) {
    if (!walk_drop(wa, sh, w)) return -1;
    walk_request(sh, w, i, j);
  }
  return walk_take(wa, sh, w);
}

// Sweeps block rows [i0, i1) from the row below (w.cur, w.n); start: the value the grid's
// first row enters column 0 with (dead: none).  On return the list holds the last row's
// output; res is set when the grid's last cell was reached.
// Recording, chunks that do not fit the list are dropped if `loose` (lost is set).  Walking
// again, WALK_MET says that a block row's list equals its record up to the constant c.
template <int KIND>
__device__ int walk_rows(const WaveArgs& wa, WalkShared* sh, Walk& w, int i0, int i1, double start,
                         double& res, WalkMode mode, WalkRecord* recs, bool loose, bool& lost,
                         double& c) {
  const int lane = threadIdx.x & 31;
  const double dead = walk_dead<KIND>();
  const int R = KIND == K_DFD ? sh->pd.n1 : sh->pd.n1 - 1;
  const int C = KIND == K_DFD ? sh->pd.n2 : sh->pd.n2 - 1;
  const int nbr = (R + 31) >> 5, nbc = (C + 31) >> 5;
  const bool flat = KIND != K_DEC && sh->flat;
  int j_min = INT_MAX, j_max = 0;
  unsigned cells = 0;
  int status = WALK_OK;
  for (int i = i0; i < i1 && status == WALK_OK; ++i) {
    const int in = w.cur, ob = w.cur ^ 1;
    const int nr = min(32, R - (i << 5));
    // the record to compare with, loaded while the row is walked
    int rec_n = -1, rec_j = 0;
    double rec_v[kWalkRec];
    if (mode == WALK_AGAIN) {
      const WalkRecord* q = recs + i;
      rec_n = __ldcg(&q->n);
      if (lane < kWalkRec) rec_j = __ldcg(&q->j[lane]);
#pragma unroll
      for (int e = 0; e < kWalkRec; ++e) rec_v[e] = __ldcg(&q->v[e][lane]);
    }
    int k = 0, on = 0, j = -1;
    unsigned bmask = 0u;  // rows that enter the next block live, values in sh->bot[bb]
    int bb = 0;
    if (i == 0 && walk_live<KIND>(start)) {
      bmask = 1u;
      j = 0;
      if (lane == 0) sh->bot[0][0] = start;
      __syncwarp();
    }
    while (status == WALK_OK) {
      if (j < 0) {
        if (k >= w.n) break;
        j = sh->up_j[in][k];
      }
      const bool have = k < w.n && sh->up_j[in][k] == j;
      const double* upv = have ? sh->up_v[in][k] : sh->dead_row;
      double F = upv[lane];
      unsigned V = __ballot_sync(kFull, walk_live<KIND>(F));
      k += have;
      // (on its way while the tile is waited for)
      const bool ask = (w.blocks & 3) == 3;
      const unsigned stop = ask && mode != WALK_ALONE ? *(volatile unsigned*)w.stop : 0u;
      const int slot = walk_get(wa, sh, w, i, j);
      if (slot < 0) { status = WALK_ERROR; break; }
      j_min = min(j_min, j);
      j_max = max(j_max, j);
      w.blocks += 1;
      w.effort += 1 + (sh->cnt[slot] >> 8);
      if (on == kWalkCap && !loose) {
        status = WALK_GIVE_UP;
        break;
      }
      if (ask) {
        const int quit =
            mode != WALK_ALONE && stop == w.sweeps ? WALK_STOPPED
            : walk_slow(w, (i - i0) + (j_max - j_min) + 1, nbr + nbc, max(on, w.n), i1 - i0, i1 - 1 - i)
                ? WALK_GIVE_UP : WALK_OK;
        status = bcast(quit);
        if (status != WALK_OK) break;
      }
      {
        // the next block: right when this one's last column has a live edge, else the next
        // chunk of the row, else up
        const uint4 m = sh->mask[slot][lane];
        const bool right = __any_sync(kFull, m.w >> 31);
        cells += __reduce_add_sync(kFull, __popc(m.x | m.y));
        const bool more = k < w.n;
        const int jn = more ? sh->up_j[in][k] : 0;
        int ni = -1, nj = 0;
        if (j + 1 < nbc && (right | (more & (jn == j + 1)))) {
          ni = i;
          nj = j + 1;
        } else if (more) {
          ni = i;
          nj = jn;
        } else if (i + 1 < i1) {
          ni = i + 1;
          nj = on ? sh->up_j[ob][0] : j;
        }
        if (ni >= 0) walk_request(sh, w, ni, nj);
      }
      unsigned omask = 0u, Y = 0u;
      const double* bin = sh->bot[bb];
      double* bout = sh->bot[bb ^ 1];
      double y = dead, f = dead;
      const int cl = (C - 1) & 31;  // the grid's last column in its block
      const bool last = i == nbr - 1 && j == nbc - 1;
      if (KIND == K_DEC || flat) {
        int r = 0, by_row = 1;
        while ((r < nr) & ((V | (r < 32 ? bmask >> r : 0u)) != 0u)) {
          const int bad = walk_bits<KIND>(sh, slot, r, nr, bmask, bin, bout, F, V, omask, Y);
          if (bad == nr) {
            r = nr;
            break;
          }
          if constexpr (KIND == K_DEC) {
            // the row that bits do not settle, with its values (the second time in a block 8
            // rows, then the rest: such rows come together)
            const int to = min(nr, bad + by_row);
            by_row <<= 3;
#pragma unroll 1
            for (r = bad; r < to; ++r) {
              walk_row(sh, slot, r, (bmask >> r) & 1u, bin[r], F, V, y, Y);
              if ((lane == 31) & (int)(Y >> 31)) bout[r] = y;
              omask |= (Y >> 31) << r;
            }
          }
        }
        if (r < nr) Y = 0u;
      } else {
        const int nc = min(32, C - (j << 5));
        // (the row handed on goes to the list at once; without room, to the row not used)
        double* out = on < kWalkCap ? sh->up_v[ob][on] : sh->spare_row;
        walk_values<KIND>(sh, slot, nr, nc, upv, V, bmask, bin, bout, omask, out, y, f);
        F = out[lane];
        V = __ballot_sync(kFull, walk_live<KIND>(F));
      }
      if (last) {
        // the last cell: VE-FD the lesser of its edges, DFD its value; the decision its right
        // edge's upper end (top edge on a transposed grid) if that edge is reached
        if (KIND == K_DEC) {
          const bool tr = sh->pd.tr != 0;
          const uint4 m = sh->mask[slot][nr - 1];
          const int2 base = sh->base[slot][nr - 1];
          const unsigned at = tr ? walk_place(base.y, m.y, cl) : walk_place(base.x, m.x, cl);
          res = ((tr ? Y : V) >> cl) & 1u ? sh->vals[slot][at].y : -2.0;
        } else if (flat) {
          res = ((Y >> cl) & 1u) | (KIND == K_VEFD ? (V >> cl) & 1u : 0u) ? 0.0 : dead;
        } else {
          res = __shfl_sync(kFull, KIND == K_VEFD ? dmin(y, f) : y, nr - 1);
        }
      }
      if (status != WALK_OK) break;
      if (V && i + 1 < nbr) {
        if (on < kWalkCap) {
          sh->up_v[ob][on][lane] = F;
          if (lane == 0) sh->up_j[ob][on] = j;
          ++on;
        } else {
          lost = true;
          w.rec_from = i + 1;  // (earlier records lead to more than what is walked on)
        }
      }
      __syncwarp();
      bmask = omask;
      bb ^= 1;
      j = omask && j + 1 < nbc ? j + 1 : -1;
    }
    w.cur = ob;
    w.n = on;
    if (status != WALK_OK) break;
    if (mode != WALK_ALONE && on && lane == 0) {
      __stcg(&recs[i].lo, sh->up_j[ob][0]);
      __stcg(&recs[i].hi, sh->up_j[ob][on - 1]);
    }
    if (mode == WALK_RECORD) {
      w.rec_end = i;
      WalkRecord* q = recs + i;
      const int n = on <= kWalkRec ? on : -1;
      if (lane == 0) __stcg(&q->n, n);
      if (lane < n) __stcg(&q->j[lane], sh->up_j[ob][lane]);
      for (int e = 0; e < n; ++e) __stcg(&q->v[e][lane], sh->up_v[ob][e][lane]);
    } else if (mode == WALK_AGAIN && i + 1 < nbr && i >= w.rec_from && i <= w.rec_end &&
               rec_n == on) {
      bool same = lane >= on || sh->up_j[ob][lane] == rec_j;
      double m = 0.0;
#pragma unroll
      for (int e = 0; e < kWalkRec; ++e) {
        if (e >= on) break;
        const double v = sh->up_v[ob][e][lane];
        if (KIND == K_DEC) same &= __double_as_longlong(v) == __double_as_longlong(rec_v[e]);
        else if (v != rec_v[e]) m = fmax(m, v);
      }
      if (KIND != K_DEC) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(kFull, m, o));
#pragma unroll
        for (int e = 0; e < kWalkRec; ++e) {
          if (e >= on) break;
          const double v = sh->up_v[ob][e][lane];
          same &= v == fmax(m, rec_v[e]) && walk_live<KIND>(v) == walk_live<KIND>(rec_v[e]);
        }
      }
      if (__all_sync(kFull, same)) {
        c = m;
        status = WALK_MET;
      }
    }
    if (on == 0) break;
  }
  if (!walk_drop(wa, sh, w)) status = WALK_ERROR;
  if (lane == 0) sh->cells += cells;
  __syncwarp();
  return status;
}

// The group of CTAs that walks a pair: `size` of them, this one is `rank`; members' reports and
// ends are at `first` + rank of the arrays.
struct WalkGroup {
  int size, rank, first;
  unsigned passed;        // barriers passed
  unsigned* arrive;       // the group's arrival count
  WalkStat* stat[2];      // by round
  WalkEnd* end[3];
};

// Barrier of the group's propagators (bounded).  All CTAs of the launch are co-resident
// (cooperative launch).  false on an error.
__device__ __forceinline__ bool walk_barrier(const WaveArgs& wa, WalkGroup& g) {
  ++g.passed;
  if (g.size == 1) return true;
  __syncwarp();
  int bad = 0;
  if ((threadIdx.x & 31) == 0) {
    __threadfence();
    atomicAdd(g.arrive, 1u);
    const unsigned want = g.passed * (unsigned)g.size;
    const long long t0 = clock64();
    for (int it = 0;; ++it) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g.arrive) : "memory");
      if (v >= want) break;
      if ((it & 15) == 15 && (ld_volatile(wa.error) || clock64() - t0 > wa.spin_cycles)) {
        atomicExch(wa.error, 1);
        bad = 1;
        break;
      }
    }
    __threadfence();
  }
  return !bcast(bad);
}

__device__ __forceinline__ void walk_save_end(const WalkShared* sh, const Walk& w, WalkEnd* e) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) __stcg(&e->n, w.n);
  if (lane < w.n) __stcg(&e->j[lane], sh->up_j[w.cur][lane]);
  for (int k = 0; k < w.n; ++k) __stcg(&e->v[k][lane], sh->up_v[w.cur][k][lane]);
}
__device__ __forceinline__ void walk_load_end(WalkShared* sh, Walk& w, const WalkEnd* e) {
  const int lane = threadIdx.x & 31;
  w.cur = 0;
  w.n = __ldcg(&e->n);
  if (lane < w.n) sh->up_j[0][lane] = __ldcg(&e->j[lane]);
  for (int k = 0; k < w.n; ++k) sh->up_v[0][k][lane] = __ldcg(&e->v[k][lane]);
  __syncwarp();
}

// The list of everything that could be live in the row below block row i, sorted by column (near
// the band of an earlier sweep, if there was one: not everything, then).
__device__ bool walk_start_row(const WaveArgs& wa, WalkShared* sh, Walk& w, int i, bool& lost) {
  const int lane = threadIdx.x & 31;
  const bool near = w.near_lo <= w.near_hi;
  if (lane == 0) {
    sh->scan_to = 1;
    sh->scan_lo = near ? w.near_lo - 2 : 0;
    sh->scan_hi = near ? w.near_hi + 2 : INT_MAX - 1;
  }
  __syncwarp();
  walk_request(sh, w, kScan, i);
  if (walk_take(wa, sh, w) < 0) return false;
  const int n = min(*(volatile int*)&sh->nup, kWalkCap);
  lost = near || *(volatile int*)&sh->lost != 0;
  const int mine = lane < n ? sh->up_j[1][lane] : INT_MAX;
  int rank = 0;
  for (int k = 0; k < n; ++k) rank += __shfl_sync(kFull, mine, k) < mine;
  if (lane < n) sh->up_j[0][rank] = mine;
  for (int k = 0; k < n; ++k) sh->up_v[0][__shfl_sync(kFull, rank, k)][lane] = sh->up_v[1][k][lane];
  w.cur = 0;
  w.n = n;
  __syncwarp();
  return true;
}

// The piece of member m by where the band of an earlier sweep ran, from the records (walk_cut_row;
// the same for both its neighbours, since no record changes meanwhile).  Members past the last
// piece only keep the number of pieces.
__device__ void walk_cut(Walk& w, const PairDesc& pd, int nbr, int nbc, int pieces, int m) {
  const int lane = threadIdx.x & 31;
  const WalkRecord* recs = (const WalkRecord*)pd.recs;
  w.cut = WalkCut{pieces, nbr, nbr};
  w.near_lo = 0;
  w.near_hi = -1;
  if (m >= pieces) return;
  const int q = m + (lane & 1);  // lane 0: this piece's start, lane 1: its end
  const int row =
      q > 0 && q < pieces
          ? walk_cut_row(q, pieces, pd.n1, nbr, nbc, [&](int i) { return __ldcg(&recs[i].hi); })
          : q > 0 ? nbr : 0;
  // (the band runs up and right, so these are in order; a long way along one row leaves pieces
  // without rows)
  w.cut.row0 = __shfl_sync(kFull, row, 0);
  w.cut.row1 = __shfl_sync(kFull, row, 1);
  if (m > 0) {
    w.near_lo = __ldcg(&recs[w.cut.row0 - 1].lo);
    w.near_hi = __ldcg(&recs[w.cut.row0 - 1].hi);
  }
}

// (a pair without room for records is one piece)
__device__ __forceinline__ int walk_pieces(const PairDesc& pd, int size, int nbr, int nbc) {
  return pd.recs ? walk_pieces(size, nbr, nbc) : 1;
}

// Options of a sweep.  flat: only whether a path survives the level (every live value 0): its
// lists meet their records as soon as the live columns do.  rounds: after so many it stops as
// WALK_UNSETTLED.
struct WalkSweep {
  bool flat;
  int rounds;
  // out: the largest of the least values the pieces end with.  No path has less if the pieces
  // started from everything that could be live (sure).
  double least;
  bool sure;
  bool band;  // the sweep found a band: the records say where it ran
};

// A whole sweep of the grid in sh->pd at a level, by the group.  Returns a WalkStatus; res: the
// DP's result (VE-FD and DFD: kFltMax when the level cuts every path; decision: -2 when
// unreachable).  Every member gets the same answer; a barrier must follow before the next sweep
// (reports, ends and records are free again once all have read them).
template <int KIND>
__device__ int walk_sweep(const WaveArgs& wa, WalkShared* sh, Walk& w, WalkGroup& g, double level,
                          double rad, double seed, WalkSweep& o, double& res) {
  const int lane = threadIdx.x & 31;
  const double dead = walk_dead<KIND>();
  const double none = KIND == K_DEC ? -2.0 : kFltMax;
  const int R = KIND == K_DFD ? sh->pd.n1 : sh->pd.n1 - 1;
  const int C = KIND == K_DFD ? sh->pd.n2 : sh->pd.n2 - 1;
  const int nbr = (R + 31) >> 5, nbc = (C + 31) >> 5;
  // (members past the last piece only keep the barriers)
  const int pieces = walk_pieces(sh->pd, g.size, nbr, nbc);
  const int m = g.rank;
  if (w.cut.pieces > 0 && w.cut.pieces != pieces) {
    // cut for a grid of other pieces: again for this one, before a record changes
    walk_cut(w, sh->pd, nbr, nbc, pieces, m);
    if (!walk_barrier(wa, g)) return WALK_ERROR;
  }
  int i0, i1;
  walk_piece(w.cut, m, pieces, nbr, &i0, &i1);
  WalkRecord* recs = reinterpret_cast<WalkRecord*>(sh->pd.recs);
  if (lane == 0) {
    sh->kind = KIND;
    sh->flat = o.flat;
    sh->level = level;
    sh->rad = rad;
  }
  sh->dead_row[lane] = dead;
  w.cur = 0;
  w.n = 0;
  w.t0 = clock64();
  w.blocks = w.effort = 0;
  w.rec_from = 0;
  w.rec_end = -1;
  double start = dead;
  if (m == 0) {
    if (KIND == K_DEC) start = 0.0;
    if (KIND == K_VEFD && seed <= level) start = o.flat ? 0.0 : seed;
    if (KIND == K_DFD) {
      // the row below the grid: 0 at column 0
      sh->up_v[0][0][lane] = lane == 0 ? 0.0 : dead;
      if (lane == 0) sh->up_j[0][0] = 0;
      w.n = 1;
    }
  }
  __syncwarp();
  res = none;
  bool lost = false;
  double c = 0.0;
  if (pieces == 1) {
    int rc = WALK_OK;
    if (m == 0) rc = walk_rows<KIND>(wa, sh, w, 0, nbr, start, res, WALK_ALONE, nullptr, false, lost, c);
    const int late = bcast(w.rule == WALK_BY_TIME && clock64() > w.deadline ? kLate : 0);
    if (g.size == 1) {
      w.late = late != 0;
      return rc;
    }
    if (rc == WALK_ERROR) return rc;
    if (m == 0 && lane == 0) {
      WalkStat* q = g.stat[0] + g.first;
      __stcg(&q->res, res);
      __stcg(&q->gave_up, (rc == WALK_GIVE_UP ? kGaveUp : 0) | late);
    }
    if (!walk_barrier(wa, g)) return WALK_ERROR;
    const WalkStat* q = g.stat[0] + g.first;
    const int up = __ldcg(&q->gave_up);
    res = __ldcg(&q->res);
    w.late = (up & kLate) != 0;
    return up & kGaveUp ? WALK_GIVE_UP : WALK_OK;
  }
  ++w.sweeps;
  const bool on = m < pieces && i0 < i1;
  WalkStat me{0.0, none, on, 0, 0, 0, 0, !on};
  auto report = [&](int round) {
    if (clock64() > w.deadline) me.gave_up |= kLate;
    if (m < pieces && lane == 0) {
      WalkStat* q = g.stat[round & 1] + g.first + m;
      __stcg(&q->c, me.c);
      __stcg(&q->res, me.res);
      __stcg(&q->changed, me.changed);
      __stcg(&q->which, me.which);
      __stcg(&q->empty, me.empty);
      __stcg(&q->part, me.part);
      __stcg(&q->gave_up, me.gave_up);
      __stcg(&q->skip, me.skip);
    }
  };
  int first_empty = 0;
  double first_res = none;
  if (on) {
    bool err = false;
    if (m > 0) err = !walk_start_row(wa, sh, w, i0, lost);
    int rc = WALK_OK;
    if (!err) rc = walk_rows<KIND>(wa, sh, w, i0, i1, start, me.res, WALK_RECORD, recs, m > 0, lost, c);
    if (err || rc == WALK_ERROR) return WALK_ERROR;
    if (rc == WALK_GIVE_UP || rc == WALK_STOPPED) {
      if (rc == WALK_GIVE_UP) me.gave_up = m == 0 ? kGaveUp : kCrowded;
      if (me.gave_up == kGaveUp) walk_stop(w);
      lost = true;  // (a start from too much: the piece is left to the rounds)
      w.n = 0;
      w.rec_end = -1;
    }
    walk_save_end(sh, w, g.end[0] + g.first + m);
    first_empty = me.empty = rc != WALK_STOPPED && w.n == 0 && i1 < nbr;
    first_res = me.res;
    me.part = lost;
    if (me.empty && (m == 0 || !lost)) walk_stop(w);
    if (KIND != K_DEC && w.rec_end >= 0) {
      // the least value the piece ends with, in place of the constant in this report
      double v = i1 == nbr ? me.res : dead;
      for (int k = 0; k < w.n; ++k) v = fmin(v, sh->up_v[w.cur][k][lane]);
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) v = fmin(v, __shfl_xor_sync(kFull, v, s));
      me.c = v < kFltMax ? v : 0.0;
    }
  }
  report(0);
  for (int round = 0;; ++round) {
    if (!walk_barrier(wa, g)) return WALK_ERROR;
    // the round's reports
    const WalkStat* st = g.stat[round & 1] + g.first;
    int moved = INT_MAX, bad = 0, hollow = INT_MAX, hollow_all = 0, part = 0, end = 0;
    int crowd = 0;  // pieces left to the rounds: 2 each, against one for each piece
    double cc = 0.0;
    for (int q = lane; q < pieces; q += 32) {
      const WalkStat* s = st + q;
      if (__ldcg(&s->skip)) continue;
      end = q;
      const int empty = __ldcg(&s->empty);
      const int up = __ldcg(&s->gave_up);
      bad |= up;
      crowd += (up & kCrowded ? 2 : 0) - 1;
      if (round > 0 && __ldcg(&s->changed)) moved = min(moved, q);
      if (empty) hollow = min(hollow, q);
      const int lossy = __ldcg(&s->part);
      part |= lossy;
      if (empty && !lossy) hollow_all = 1;
      cc = fmax(cc, __ldcg(&s->c));
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      moved = min(moved, __shfl_xor_sync(kFull, moved, d));
      hollow = min(hollow, __shfl_xor_sync(kFull, hollow, d));
      bad |= __shfl_xor_sync(kFull, bad, d);
      crowd += __shfl_xor_sync(kFull, crowd, d);
      hollow_all |= __shfl_xor_sync(kFull, hollow_all, d);
      part |= __shfl_xor_sync(kFull, part, d);
      end = max(end, __shfl_xor_sync(kFull, end, d));
      cc = fmax(cc, __shfl_xor_sync(kFull, cc, d));
    }
    const double last = __ldcg(&st[end].res);
    int done = 0, rc = WALK_OK;
    w.late = (bad & kLate) != 0;
    if (bad & kGaveUp) {
      done = 1;
      rc = WALK_GIVE_UP;
    } else if (round == 0) {
      // a walk from everything that could be live died: so does the sweep
      done = hollow_all || hollow == 0;
      o.least = cc;
      o.sure = !part;
      me.c = 0.0;
    } else if (moved == INT_MAX) {
      // every piece was walked from its predecessor's end: the ends are the true ones
      done = 1;
      if (hollow == INT_MAX) res = (KIND == K_DEC || !(last < kFltMax)) ? last : fmax(cc, last);
    } else {
      done = hollow <= moved;  // (ends up to the first that moved are the true ones)
    }
    if (!done && round >= o.rounds) {
      done = 1;
      rc = WALK_UNSETTLED;
    }
    // (of more than half of the pieces left to the rounds some follow one another)
    if ((!done || rc == WALK_UNSETTLED) && (w.late || (w.pace > 0.f && round == 0 && crowd > 0))) {
      done = 1;
      rc = WALK_GIVE_UP;
    }
    int from = 0, again = 0;
    int before = m - 1;  // the piece below this one
    if (!done && on && m > 0) {
      while (before > 0 && __ldcg(&st[before].skip)) --before;
      again = round == 0 || __ldcg(&st[before].changed);
      from = __ldcg(&st[before].which);
    }
    if (done && rc == WALK_OK && res != none) {
      walk_cut(w, sh->pd, nbr, nbc, pieces, m);
      o.band = true;
    }
    if (done) return rc;
    const int was = me.which;
    me.changed = 0;
    if (again) {
      walk_load_end(sh, w, g.end[from] + g.first + before);
      w.t0 = clock64();
      w.blocks = w.effort = 0;
      c = 0.0;
      double r = none;
      int q = WALK_OK;
      if (w.n) q = walk_rows<KIND>(wa, sh, w, i0, i1, dead, r, WALK_AGAIN, recs, false, lost, c);
      if (q == WALK_ERROR) return WALK_ERROR;
      me.gave_up = q == WALK_GIVE_UP ? kGaveUp : 0;
      if (me.gave_up) walk_stop(w);
      if (q == WALK_MET) {
        me.which = 0;
        me.c = c;
        me.res = first_res;
        me.empty = first_empty;
        me.changed = was != 0;
      } else {
        me.which = was == 1 ? 2 : 1;
        me.c = 0.0;
        me.res = r;
        me.empty = w.n == 0 && i1 < nbr;
        me.changed = 1;
        walk_save_end(sh, w, g.end[me.which] + g.first + m);
      }
    }
    report(round + 1);
  }
}

// The value of a min-max DP, by the group, or kFltMax if it exceeds the level (a WalkStatus is
// returned).  Where the pieces' values do not meet their records within a few rounds (a wide band
// keeps the values of its start apart, though its live columns soon agree), the least value a
// path can have is guessed from the pieces' ends and settled by flat sweeps: some path survives
// it, and none survives the next smaller number.
template <int KIND>
__device__ int walk_value(const WaveArgs& wa, WalkShared* sh, Walk& w, WalkGroup& g, double level,
                          double seed, bool& band, double& res) {
  constexpr int kRounds = 3;
  int rc = WALK_OK;
  // one sweep and the barrier after it; true when the caller goes on with `out`
  double out = kFltMax;
  WalkSweep o{false, kRounds, 0.0, false, false};
  auto sweep = [&](bool flat, int rounds, double at) -> bool {
    rc = WALK_GIVE_UP;
    if (w.late) return false;
    o.flat = flat;
    o.rounds = rounds;
    rc = walk_sweep<KIND>(wa, sh, w, g, at, sqrt(at), seed, o, out);
    band |= o.band;
    if (!walk_barrier(wa, g)) rc = WALK_ERROR;
    return rc == WALK_OK;
  };
  // flat sweeps around a candidate: 1 it is the value, 0 it is not, -1 error or given up
  auto settles = [&](double x, bool sure) -> int {
    if (!sweep(true, INT_MAX, x)) return -1;
    if (!(out < kFltMax)) return 0;
    if (sure || x == 0.0) return 1;
    if (!sweep(true, INT_MAX, __longlong_as_double(__double_as_longlong(x) - 1))) return -1;
    return out < kFltMax ? 0 : 1;
  };
  for (int turn = 0;; ++turn) {
    if (sweep(false, turn < 2 ? kRounds : INT_MAX, level)) {
      res = out;
      return WALK_OK;
    }
    if (rc != WALK_UNSETTLED) return rc;
    const double x = o.least;
    const int s = settles(x, o.sure);
    if (s < 0) return rc;
    if (s == 1) {
      res = x;
      return WALK_OK;
    }
    // does any path survive the level?  (If so, the next turn's pieces start near it.)
    if (!sweep(true, INT_MAX, level)) return rc;
    if (!(out < kFltMax)) {
      res = kFltMax;
      return WALK_OK;
    }
  }
}

}  // namespace rfd
