// dndsg_lusgs.cuh -- the scan-order LU-SGS sweep on the GPU (UpdateLUSGSForward / UpdateLUSGSBackward,
// DNDS_FV_EulerEvaluator.cpp:1149-1357): a parallel pass that writes one record per schedule position,
// and the sequential walk over the records (schedule: dndsg_lusgs_sched.hpp).
#pragma once
#include "dndsg_async.cuh"
#include "dndsg_bodies.cuh"
#include "dndsg_lusgs_sched.hpp"
#include "dndsg_sa.cuh"

namespace dg {

// The neighbour term of a sweep, w (dF(U_j; n, dU_j) - lam dU_j) (fluxJacobian0_Right_Times_du,
// DNDS_FV_EulerEvaluator.hpp:928-956), is linear in the neighbour's increment and everything else in it is
// fixed during the sweep, so a cell's update is
//   dU_i = x0 + sum_q M_q dU_q,   x0 = D^-1 rhs (forward) or the forward increment (backward),
// with the 4x4 matrices M_q (times D^-1) of its up to 4 used neighbours.  U5 of an SA context adds one row
// per neighbour over (dU0, dU1, dU2, dU5).
//
// What bounds the walk is the latency of one level (a level needs the one before it), so the record
// holds finished matrix rows: four lanes compute a cell, each one row, a chain of two products and three
// sums per level.  Records with the generating quantities of a matrix (10 values instead of 16) made that
// chain 15 operations and one thread's work per cell, and the copying of the records, in step with every
// level, took longer than the level: 0.6-0.7 us.  Now 0.23-0.30 us per level: in natural order on 512 x 128 quads with
// U5, 639 levels, 482 -> 172 us forward and 464 -> 194 us backward (three neighbours per record, at the wake cut), on
// 256 x 64 quads, 319 levels, 203 -> 74 and 80 us, in 16 parts of the former, 159 levels, 97 -> 40 us.

// the fields of a context that the records are made of
struct WalkGeom {
  int64_t n;
  const double *u, *vol, *faceArea, *faceNormal, *lamA;
  double gamma;
};
struct WalkDev {  // a WalkSchedule on the device
  const int32_t *nbF, *nbJ;
  const WalkMeta* meta;
  const WalkBatch* batches;
  const int32_t* blockBatch;
  int K, mail, bars;
};

// the records of one sweep, four lanes per schedule position (lane v: row v), so that a position's
// rows leave as whole 128-byte lines.  A neighbour in another part (backward sweeps) is a ghost with its
// increment after the forward sweep, which inc holds while this kernel runs: its term goes into x0.
template <int NS, bool FWD, bool SA>
__global__ void __launch_bounds__(256) k_lusgs_records(WalkGeom g, WalkDev sc, double alpha, const double* Dinv,
                                                       const double* rhs, const double* inc, const double* u5,
                                                       const double* Dinv5, const double* rhs5, const double* inc5,
                                                       unsigned char* rec, unsigned char* rec5) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t t = e >> 2;
  const int v = (int)(e & 3);
  if (t >= g.n) return;
  const int4 f4 = reinterpret_cast<const int4*>(sc.nbF)[t], j4 = reinterpret_cast<const int4*>(sc.nbJ)[t];
  const int32_t fa[4] = {f4.x, f4.y, f4.z, f4.w}, ja[4] = {j4.x, j4.y, j4.z, j4.w};
  unsigned char* r = rec + t * walk_rec_bytes(NS);
  unsigned char* r5 = SA ? rec5 + t * walk_rec5_bytes(NS) : nullptr;
  if (v < 2)
    reinterpret_cast<int4*>(r + NS * 128 + 32)[v] = reinterpret_cast<const int4*>(sc.meta + t)[v];
  const int64_t i = sc.meta[t].cell;
  const double di = Dinv[i], di5 = SA ? Dinv5[i] : 0.0, g1 = g.gamma - 1;
  const double scale = -0.5 * alpha / g.vol[i];
  double x0 = FWD ? di * rhs[4 * i + v] : inc[4 * i + v];
  double x5 = 0.0;
  if (SA && v == 0) x5 = FWD ? di5 * rhs5[i] : inc5[i];
  int nu = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (ja[k] == -1) continue;
    const bool ghost = ja[k] < 0;
    const int64_t j = ghost ? kWalkGhost - ja[k] : ja[k];
    const int32_t f = fa[k] >= 0 ? fa[k] : ~fa[k];
    const double sg = fa[k] >= 0 ? 1.0 : -1.0, area = g.faceArea[f];
    const double nx = sg * g.faceNormal[2 * (int64_t)f], ny = sg * g.faceNormal[2 * (int64_t)f + 1];
    const double w = scale * area, wl = w * (g.lamA[f] / area);
    double U[4];
    load4<double>(&g.u[4 * j], U);
    const double ir = 1.0 / U[0];
    const double vx = U[1] * ir, vy = U[2] * ir, q2 = vx * vx + vy * vy, kq = 0.5 * q2;
    const double p = g1 * (U[3] - 0.5 * U[0] * q2), H = (U[3] + p) * ir, vn = vx * nx + vy * ny;
    // row v of w dF - wl dU: with a = nx dU1 + ny dU2 - vn dU0 and dp = g1 (dU3 - vx dU1 - vy dU2 + kq dU0),
    //   dF = (nx dU1 + ny dU2, vn dU1 + vx a + nx dp, vn dU2 + vy a + ny dp, H a + vn (dU3 + dp))
    const double ca = v == 0 ? 1.0 : (v == 1 ? vx : (v == 2 ? vy : H));             // factor of a (row 0: a + vn dU0)
    const double cp = g1 * (v == 0 ? 0.0 : (v == 1 ? nx : (v == 2 ? ny : vn)));     // factor of dp / g1
    const double cv = v == 0 ? vn : 0.0;
    double m[4] = {cp * kq - ca * vn + cv, ca * nx - cp * vx, ca * ny - cp * vy, cp};
    m[v == 0 ? 0 : v] += v == 0 ? 0.0 : vn;
    for (int c = 0; c < 4; c++) m[c] = w * m[c] - (c == v ? wl : 0.0);
    const double c5 = SA && v == 0 ? w * u5[j] * ir : 0.0;
    if (!FWD && ghost) {
      double d[4];
      load4<double>(&inc[4 * j], d);
      x0 += di * (m[0] * d[0] + m[1] * d[1] + m[2] * d[2] + m[3] * d[3]);
      if (SA && v == 0) x5 += di5 * (c5 * (nx * d[1] + ny * d[2] - vn * d[0]) + (w * vn - wl) * inc5[j]);
      continue;
    }
    double2* o = reinterpret_cast<double2*>(r + nu * 128 + v * 16);
    o[0] = make_double2(di * m[0], di * m[1]);
    o[4] = make_double2(di * m[2], di * m[3]);
    if (SA && v == 0) {
      double2* o5 = reinterpret_cast<double2*>(r5 + nu * 32);
      o5[0] = make_double2(-di5 * c5 * vn, di5 * c5 * nx);
      o5[1] = make_double2(di5 * c5 * ny, di5 * (w * vn - wl));
    }
    nu++;
  }
  for (; nu < NS; nu++) {
    double2* o = reinterpret_cast<double2*>(r + nu * 128 + v * 16);
    o[0] = o[4] = make_double2(0.0, 0.0);
    if (SA && v == 0) {
      double2* o5 = reinterpret_cast<double2*>(r5 + nu * 32);
      o5[0] = o5[1] = make_double2(0.0, 0.0);
    }
  }
  *reinterpret_cast<double*>(r + NS * 128 + 8 * v) = x0;
  if (SA && v == 0) *reinterpret_cast<double2*>(r5 + NS * 32) = make_double2(x5, 0.0);
}

__device__ __forceinline__ double2 lds2(uint32_t a) {
  double2 r;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(r.x), "=d"(r.y) : "r"(a) : "memory");
  return r;
}
__device__ __forceinline__ double lds1(uint32_t a) {
  double r;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r) : "r"(a) : "memory");
  return r;
}
__device__ __forceinline__ int4 lds_i4(uint32_t a) {
  int4 r;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a) : "memory");
  return r;
}
__device__ __forceinline__ void sts1(uint32_t a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }

// A copying warp (w of kWalkCopy) of a walk: every kWalkCopy-th batch's records into its stage.  Returns its last
// batch; failed: a wait ran out.
template <int RB, int RB5, int S, int W>
__device__ __forceinline__ int walk_copy(int w, int lane, int32_t nb, const WalkBatch* bat, const unsigned char* rec,
                                         const unsigned char* rec5, uint32_t full, uint32_t empty, uint32_t stR, uint32_t stR5,
                                         bool& failed) {
  int last = -1;
  int32_t first = 0, cnt = 0;  // lane k keeps the first positions of the warp's k-th next batches
  for (int l = w, k = 0; l < nb; l += kWalkCopy, k = (k + 1) & 31) {
    if (k == 0) {
      const WalkBatch x = bat[min(l + kWalkCopy * lane, nb - 1)];
      first = x.first;
      cnt = x.n;
    }
    const int32_t a = __shfl_sync(0xffffffffu, first, k), n = __shfl_sync(0xffffffffu, cnt, k);
    const uint32_t st = (uint32_t)(l % S), bar = full + 8 * st;
    const bool ok = l < S || mbar_wait(empty + 8 * st, (uint32_t)(l / S - 1) & 1u, kWaitLimit);
    failed = __any_sync(0xffffffffu, !ok);
    if (failed) break;
    if (lane == 0) {
      mbar_expect_tx(bar, (uint32_t)(n * (RB + RB5)));
      bulk_g2s(stR + st * W * RB, rec + (int64_t)a * RB, (uint32_t)(n * RB), bar);
      if (RB5) bulk_g2s(stR5 + st * W * RB5, rec5 + (int64_t)a * RB5, (uint32_t)(n * RB5), bar);
    }
    last = l;
  }
  return last;
}
// After a timeout: the warp's copies in flight land before the block leaves.  A stage's phase may never complete then
// (the mailbox warp or a computing warp left its part out), so these waits are short against kWaitLimit and long
// against a copy, or an increment on its way between two blocks
constexpr uint32_t kWalkDrain = 1u << 14;
template <int S>
__device__ __forceinline__ void walk_drain(int last, uint32_t full) {
  for (int l = max(last - S + kWalkCopy, 0); l <= last; l++)
    if (l % kWalkCopy == last % kWalkCopy) mbar_wait(full + 8 * (l % S), (uint32_t)(l / S) & 1u, kWalkDrain);
}

// The mailbox warp of a cluster's block: a batch's stage is full once its records are there and, by this warp, the
// increments that it is the first to need.  The wait acquires at cluster scope, which takes longer than a wait at the
// block's own: in the computing warps it was on the way of every level (natural order, RANS-SA on 512 x 128 cells 745 us
// an iteration, laminar flow with GMRES on 256 x 64 cells 7.91 ms; by this warp 656 us and 6.63 ms).
template <int S>
__device__ __forceinline__ void walk_mail(int lane, int32_t nb, const WalkBatch* bat, uint32_t full, uint32_t empty, uint32_t mailB,
                                          bool& failed) {
  int32_t bars = -1, next = lane < nb ? bat[lane].bar : -1;  // lane k: batch l + k's barrier
  for (int l = 0; l < nb; l++) {
    if ((l & 31) == 0) {
      bars = next;
      next = l + 32 + lane < nb ? bat[l + 32 + lane].bar : -1;
    }
    const int32_t bar = __shfl_sync(0xffffffffu, bars, l & 31);
    const uint32_t st = (uint32_t)(l % S);
    bool ok = l < S || mbar_wait(empty + 8 * st, (uint32_t)(l / S - 1) & 1u, kWaitLimit);
    if (ok && bar >= 0) ok = mbar_wait_cluster(mailB + 8 * bar, 0, kWaitLimit);
    failed = __any_sync(0xffffffffu, !ok);
    if (failed) break;
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full + 8 * st) : "memory");
  }
}

// The walk, one block per run of scan positions or cells, K blocks per part in a cluster.  Two sets of warps take the
// batches in turn.  Of a set, warps 0-3 hold row v = lane & 3 of position 8 warp + lane / 4; SA: one warp
// more, U5 of position `lane`.  A set loads its next records into registers while the other one
// computes, so that a level is on its critical path only with the increments from shared memory, the row
// product, the store and the barrier between the sets (the set that finished batch l arrives, the one that
// takes l + 1 waits).  An increment for another block goes by st.async, which completes a barrier of the
// batch that needs it there: no fence, and the mailbox warp waits for it beside the sets.  The copying warps
// keep walk_stages() batches of records in flight (two of them: one's round per batch took longer than a level,
// 0.29 against 0.22 us).  A wait that runs out sets kFlagTimeout; its warp then skips the rest of its work, keeps
// to every barrier, and the blocks leave together (a mailbox may be written until its block's peers are done, and
// a little later for one whose own waits did not see the last increments come).
template <int NS, bool SA>
__global__ void __launch_bounds__(walk_threads(SA, kWalkW), 1) k_lusgs_walk(WalkDev sc, const unsigned char* rec,
                                                                    const unsigned char* rec5, double* inc, double* inc5,
                                                                    unsigned* flags) {
  extern __shared__ __align__(128) unsigned char sm[];
  constexpr int RB = walk_rec_bytes(NS), RB5 = SA ? walk_rec5_bytes(NS) : 0;
  constexpr int S = walk_stages(kWalkW), NW = walk_rows(SA) / 32;  // warps of a set
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = sc.K, nval = kWalkZero + 1 + sc.mail;
  const uint32_t full = smem_u32(sm), empty = full + 8 * S, mailB = full + 16 * S, vals = mailB + ((sc.bars * 8 + 31) & ~31),
                 vals5 = vals + nval * 32;
  const uint32_t stR = vals5 + (SA ? ((nval * 8 + 15) & ~15) : 0), stR5 = stR + S * kWalkW * RB;
  const int32_t b0 = sc.blockBatch[blockIdx.x], nb = sc.blockBatch[blockIdx.x + 1] - b0;
  const WalkBatch* bat = sc.batches + b0;
  if (tid == 0)
    for (int k = 0; k < S; k++) {
      mbar_init(full + 8 * k, K > 1 ? 2 : 1);
      mbar_init(empty + 8 * k, NW);
    }
  if (K > 1)
    for (int l = tid; l < nb; l += blockDim.x) {
      const WalkBatch x = bat[l];
      if (x.bar >= 0) mbar_init(mailB + 8 * x.bar, 1);
    }
  fence_mbar_init();
  if (K > 1)  // every mailbox barrier: one phase, complete when its slots' bytes are in
    for (int l = tid; l < nb; l += blockDim.x) {
      const WalkBatch x = bat[l];
      if (x.bar >= 0) mbar_expect_tx(mailB + 8 * x.bar, (uint32_t)(x.slots * (SA ? 40 : 32)));
    }
  if (tid < 4) sts1(vals + kWalkZero * 32 + 8 * tid, 0.0);
  if (SA && tid == 4) sts1(vals5 + kWalkZero * 8, 0.0);
  __syncthreads();
  if (K > 1) cluster_sync_all();
  bool failed = false;
  int last = -1;  // the copying warp's last batch
  if (warp == 2 * NW + kWalkCopy) {
    if (K > 1) walk_mail<S>(lane, nb, bat, full, empty, mailB, failed);
  } else if (warp >= 2 * NW) {
    last = walk_copy<RB, RB5, S, kWalkW>(warp - 2 * NW, lane, nb, bat, rec, rec5, full, empty, stR, stR5, failed);
  } else {
    const int set = warp >= NW ? 1 : 0, sw = warp - set * NW;
    const bool rows = sw < 4;
    const int32_t p0 = nb > 0 ? bat[0].first : 0;
    const int pos = rows ? sw * 8 + (lane >> 2) : lane, v = lane & 3;
    const uint32_t myRec = stR + pos * RB, myRow = rows ? myRec + v * 16 : stR5 + pos * RB5,
                   myX0 = rows ? myRec + NS * 128 + 8 * v : myRow + NS * 32;
    constexpr int kSets = 2 * walk_rows(SA);  // threads of both sets, which the barriers 1 and 2 count
    int4 bt = set < nb ? *reinterpret_cast<const int4*>(bat + set) : make_int4(0, 0, -1, 0);
    for (int l = set; l < nb; l += 2) {
      // ---- beside the other set's batch: the records of this one
      const uint32_t st = (uint32_t)(l % S), o = st * (rows ? kWalkW * RB : kWalkW * RB5), r = myRec + st * kWalkW * RB;
      const int4 cur = bt;  // first position, positions
      if (l + 2 < nb) bt = *reinterpret_cast<const int4*>(bat + l + 2);
      if (!failed) failed = !mbar_wait(full + 8 * st, (uint32_t)(l / S) & 1u, kWaitLimit);
      // (lanes past the batch's positions read stale data and drop it)
      const int4 src4 = lds_i4(r + NS * 128 + 32), to = lds_i4(r + NS * 128 + 48);
      double2 m[NS][2];
#pragma unroll
      for (int q = 0; q < NS; q++) {
        m[q][0] = lds2(myRow + o + (rows ? q * 128 : q * 32));
        m[q][1] = lds2(myRow + o + (rows ? q * 128 + 64 : q * 32 + 16));
      }
      const double x0 = lds1(myX0 + o);
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * st) : "memory");
      const bool act = pos < cur.y && !failed;
      const int32_t sr[4] = {src4.x, src4.y, src4.z, src4.w}, push[kWalkPush] = {to.x, to.y, to.z};
      uint32_t at[NS], pushAt[kWalkPush], pushBar[kWalkPush];
      bool old = false;
#pragma unroll
      for (int q = 0; q < NS; q++) {
        at[q] = vals + (uint32_t)(sr[q] < 0 ? kWalkZero * 32 : sr[q]);
        old = old || sr[q] < 0;
      }
      if (K > 1 && act) {
#pragma unroll
        for (int q = 0; q < kWalkPush; q++) {
          if (push[q] < 0) break;
          const uint32_t x = (uint32_t)push[q], blk = x >> (2 * kWalkSlotBits), sl = kWalkZero + 1 + (x & kWalkMaxMail);
          pushAt[q] = cluster_map(rows ? vals + sl * 32 + 8 * v : vals5 + sl * 8, blk);
          pushBar[q] = cluster_map(mailB + 8 * (x >> kWalkSlotBits & kWalkMaxMail), blk);
        }
      }
      const uint32_t slot = (uint32_t)(cur.x + pos - p0) & (kWalkRing - 1);
      const uint32_t mine = rows ? vals + slot * 32 + 8 * v : vals5 + slot * 8;
      // ---- batch l - 1 is finished
      if (l > 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + ((l - 1) & 1)), "n"(kSets) : "memory");
      double a = x0;
      if (act) {
        double2 d[NS][2];
#pragma unroll
        for (int q = 0; q < NS; q++) {
          d[q][0] = lds2(at[q]);
          if (SA && !rows) d[q][1] = make_double2(lds1(at[q] + 16), lds1(vals5 + ((at[q] - vals) >> 2)));
          else d[q][1] = lds2(at[q] + 16);
        }
        if (old) {
#pragma unroll
          for (int q = 0; q < NS; q++)
            if (sr[q] < 0) {  // a position of this block that left the ring, stored before an earlier barrier
              const int64_t j = -(int64_t)sr[q] - 1;
              d[q][0] = *reinterpret_cast<const double2*>(&inc[4 * j]);
              // (one load for both and the U5 value over it would make the U5 warp wait once per neighbour)
              if (SA && !rows) d[q][1] = make_double2(inc[4 * j + 2], inc5[j]);
              else d[q][1] = *reinterpret_cast<const double2*>(&inc[4 * j + 2]);
            }
        }
        double b = 0.0;
#pragma unroll
        for (int q = 0; q < NS; q++) {
          const double s0 = fma(m[q][0].y, d[q][0].y, m[q][0].x * d[q][0].x);
          const double s1 = fma(m[q][1].y, d[q][1].y, m[q][1].x * d[q][1].x);
          if (q & 1) b += s0 + s1;
          else a += s0 + s1;
        }
        a += b;
        sts1(mine, a);
        if (K > 1) {
#pragma unroll
          for (int q = 0; q < kWalkPush; q++) {
            if (push[q] < 0) break;
            st_async_f64(pushAt[q], a, pushBar[q]);
          }
        }
      }
      asm volatile("bar.arrive %0, %1;" ::"r"(1 + (l & 1)), "n"(kSets) : "memory");
      // the increment itself: read from there only once its position has left the ring, at least
      // kWalkRing / kWalkW - 1 batches and as many barriers on
      if (act) {
        if (rows) inc[4 * (int64_t)to.w + v] = a;
        else inc5[to.w] = a;
      }
    }
    if (nb > 0 && set == (nb & 1))  // the set that did not take the last batch
      asm volatile("bar.sync %0, %1;" ::"r"(1 + ((nb - 1) & 1)), "n"(kSets) : "memory");
  }
  if (failed) atomicOr(flags, kFlagTimeout);
  __syncwarp();
  const bool any = __syncthreads_or(failed);
  if (any && lane == 0) walk_drain<S>(last, full);
  if (K > 1) {
    __syncwarp();
    cluster_sync_all();  // no increment is sent after this
    if (any)  // those on their way here land before the block leaves; the ones that a failed warp left out never do
      for (int l = tid; l < nb; l += blockDim.x) {
        const WalkBatch x = bat[l];
        if (x.bar >= 0) mbar_wait_cluster(mailB + 8 * x.bar, 0, kWalkDrain);
      }
  }
}

// The walk of parts of one block with wide levels: batches of kWalkWide positions, two of them (32 apart) in every
// lane.  There the latency of a set's own round (its records into registers, the increments, the store) bounds the
// walk, and two positions share it: sweeps in one block of 512 x 128 quads in natural order, levels of 103 cells, 462 ->
// 315 us, of 256 x 64, levels of 51, 127 -> 91 us; of 262,144 quads numbered at random 4,035 -> 3,160 us (65,536 with
// U5: the iteration 2,830 -> 2,494 us); 75 parts of 112 x 224 quads 538 -> 498 us.  An increment that left the ring was
// stored at least four batches and as many barriers before.
template <int NS, bool SA>
__global__ void __launch_bounds__(walk_threads(SA, kWalkWide), 1) k_lusgs_walk_wide(WalkDev sc, const unsigned char* rec,
                                                                                   const unsigned char* rec5, double* inc,
                                                                                   double* inc5, unsigned* flags) {
  extern __shared__ __align__(128) unsigned char sm[];
  constexpr int RB = walk_rec_bytes(NS), RB5 = SA ? walk_rec5_bytes(NS) : 0;
  constexpr int W = kWalkWide, S = walk_stages(W), NW = walk_rows(SA) / 32, R = W / 32;  // NW: warps of a set
  constexpr int nval = kWalkZero + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full = smem_u32(sm), empty = full + 8 * S, vals = full + 16 * S, vals5 = vals + nval * 32;
  const uint32_t stR = vals5 + (SA ? ((nval * 8 + 15) & ~15) : 0), stR5 = stR + S * W * RB;
  const int32_t b0 = sc.blockBatch[blockIdx.x], nb = sc.blockBatch[blockIdx.x + 1] - b0;
  const WalkBatch* bat = sc.batches + b0;
  if (tid == 0)
    for (int k = 0; k < S; k++) {
      mbar_init(full + 8 * k, 1);
      mbar_init(empty + 8 * k, NW);
    }
  fence_mbar_init();
  if (tid < 4) sts1(vals + kWalkZero * 32 + 8 * tid, 0.0);
  if (SA && tid == 4) sts1(vals5 + kWalkZero * 8, 0.0);
  __syncthreads();
  bool failed = false;
  int last = -1;
  if (warp >= 2 * NW) {
    last = walk_copy<RB, RB5, S, W>(warp - 2 * NW, lane, nb, bat, rec, rec5, full, empty, stR, stR5, failed);
  } else {
    const int set = warp >= NW ? 1 : 0, sw = warp - set * NW;
    const bool rows = sw < 4;
    const int32_t p0 = nb > 0 ? bat[0].first : 0;
    const int v = lane & 3;
    const int pos = rows ? sw * 8 + (lane >> 2) : lane;  // and 32 more
    const uint32_t myRec = stR + pos * RB, myRow = rows ? myRec + v * 16 : stR5 + pos * RB5,
                   myX0 = rows ? myRec + NS * 128 + 8 * v : myRow + NS * 32;
    constexpr int kSets = 2 * walk_rows(SA);  // threads of both sets, which the barriers 1 and 2 count
    int4 bt = set < nb ? *reinterpret_cast<const int4*>(bat + set) : make_int4(0, 0, -1, 0);
    for (int l = set; l < nb; l += 2) {
      // ---- beside the other set's batch: the records of this one
      const uint32_t st = (uint32_t)(l % S), o = st * (rows ? W * RB : W * RB5);
      const int4 cur = bt;  // first position, positions
      if (l + 2 < nb) bt = *reinterpret_cast<const int4*>(bat + l + 2);
      if (!failed) failed = !mbar_wait(full + 8 * st, (uint32_t)(l / S) & 1u, kWaitLimit);
      // (lanes past the batch's positions read stale data and drop it)
      int4 src4[R];
      int32_t cell[R];
      double2 m[R][NS][2];
      double x0[R];
#pragma unroll
      for (int e = 0; e < R; e++) {
        const uint32_t r = myRec + (st * W + 32 * e) * RB, y = o + 32 * e * (rows ? RB : RB5);
        src4[e] = lds_i4(r + NS * 128 + 32);
        cell[e] = lds_i4(r + NS * 128 + 48).w;
#pragma unroll
        for (int q = 0; q < NS; q++) {
          m[e][q][0] = lds2(myRow + y + (rows ? q * 128 : q * 32));
          m[e][q][1] = lds2(myRow + y + (rows ? q * 128 + 64 : q * 32 + 16));
        }
        x0[e] = lds1(myX0 + y);
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * st) : "memory");
      bool act[R], old = false;
      uint32_t at[R][NS], mine[R];
#pragma unroll
      for (int e = 0; e < R; e++) {
        act[e] = pos + 32 * e < cur.y && !failed;
        const int32_t sr[4] = {src4[e].x, src4[e].y, src4[e].z, src4[e].w};
#pragma unroll
        for (int q = 0; q < NS; q++) {
          at[e][q] = vals + (uint32_t)(sr[q] < 0 || !act[e] ? kWalkZero * 32 : sr[q]);
          old = old || (sr[q] < 0 && act[e]);
        }
        const uint32_t slot = (uint32_t)(cur.x + pos + 32 * e - p0) & (kWalkRing - 1);
        mine[e] = rows ? vals + slot * 32 + 8 * v : vals5 + slot * 8;
      }
      // ---- batch l - 1 is finished
      if (l > 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + ((l - 1) & 1)), "n"(kSets) : "memory");
      double2 d[R][NS][2];
#pragma unroll
      for (int e = 0; e < R; e++)
#pragma unroll
        for (int q = 0; q < NS; q++) {
          d[e][q][0] = lds2(at[e][q]);
          if (SA && !rows) d[e][q][1] = make_double2(lds1(at[e][q] + 16), lds1(vals5 + ((at[e][q] - vals) >> 2)));
          else d[e][q][1] = lds2(at[e][q] + 16);
        }
      if (old) {
#pragma unroll
        for (int e = 0; e < R; e++) {
          const int32_t sr[4] = {src4[e].x, src4[e].y, src4[e].z, src4[e].w};
#pragma unroll
          for (int q = 0; q < NS; q++)
            if (act[e] && sr[q] < 0) {
              const int64_t j = -(int64_t)sr[q] - 1;
              d[e][q][0] = *reinterpret_cast<const double2*>(&inc[4 * j]);
              if (SA && !rows) d[e][q][1] = make_double2(inc[4 * j + 2], inc5[j]);
              else d[e][q][1] = *reinterpret_cast<const double2*>(&inc[4 * j + 2]);
            }
        }
      }
      double a[R];
#pragma unroll
      for (int e = 0; e < R; e++) {
        double b = 0.0;
        a[e] = x0[e];
#pragma unroll
        for (int q = 0; q < NS; q++) {
          const double s0 = fma(m[e][q][0].y, d[e][q][0].y, m[e][q][0].x * d[e][q][0].x);
          const double s1 = fma(m[e][q][1].y, d[e][q][1].y, m[e][q][1].x * d[e][q][1].x);
          if (q & 1) b += s0 + s1;
          else a[e] += s0 + s1;
        }
        a[e] += b;
      }
#pragma unroll
      for (int e = 0; e < R; e++)
        if (act[e]) sts1(mine[e], a[e]);
      asm volatile("bar.arrive %0, %1;" ::"r"(1 + (l & 1)), "n"(kSets) : "memory");
#pragma unroll
      for (int e = 0; e < R; e++)
        if (act[e]) {
          if (rows) inc[4 * (int64_t)cell[e] + v] = a[e];
          else inc5[cell[e]] = a[e];
        }
    }
    if (nb > 0 && set == (nb & 1))  // the set that did not take the last batch
      asm volatile("bar.sync %0, %1;" ::"r"(1 + ((nb - 1) & 1)), "n"(kSets) : "memory");
  }
  if (failed) atomicOr(flags, kFlagTimeout);
  __syncwarp();
  if (__syncthreads_or(failed) && lane == 0) walk_drain<S>(last, full);
}

}  // namespace dg
