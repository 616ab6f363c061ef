// dndsg_lusgs_sched.hpp -- host side of the scan-order LU-SGS sweep: which thread block walks which cells
// in which order, and where every neighbour's increment is when a cell needs it.  Plain C++, so that the
// schedule can be checked on the CPU.
//
// A sweep in scan order is a chain of dependency levels (a cell's level is one more than the largest
// level of its earlier neighbours).  Each part (the reference's rank) is cut into K runs of consecutive
// scan positions, one thread block per run, the K blocks of a part being one thread-block cluster.  A
// block walks its own cells level by level in batches of at most kWalkW cells, a block barrier between
// batches.  Dependencies go from lower runs to higher ones in the forward sweep and the other way in the
// backward one, so the blocks never wait on one another in a circle.  A neighbour's increment is read from
//   * a ring of the block's own last kWalkRing positions (shared memory),
//   * the block's mailbox (shared memory), one slot per cell of another run that it needs: the block that
//     computes the cell stores it there over distributed shared memory, signalling a barrier of the batch that
//     needs it first (that batch waits until all its slots are filled),
//   * or, for an older position of its own, global memory.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace dg {

constexpr int kWalkW = 32;      // cells per batch: 4 lanes each, four warps
constexpr int kWalkRing = 256;  // positions in the ring (a power of two)
constexpr int kWalkMaxK = 16;   // blocks per part (one cluster)
constexpr int kWalkZero = kWalkRing;
constexpr int kWalkPush = 3;    // mailboxes that one cell's increment can go to
constexpr int kWalkSlotBits = 13, kWalkMaxMail = (1 << kWalkSlotBits) - 1;
// a mailbox and its barrier as one non-negative number: block of the part, barrier, slot
inline int32_t walk_push(int block, int bar, int slot) { return (block << (2 * kWalkSlotBits)) | (bar << kWalkSlotBits) | slot; }

// per schedule position, 32 bytes, copied into its record:
//   src[4]   where the increment of used neighbour q is: 32 times a slot of the block's shared values (ring
//            slot; kWalkZero, which holds zeros, for an unused one; kWalkZero + 1 + mailbox slot), or
//            -(j + 1): cell j in global memory
//   push[3]  walk_push of a mailbox, or -1
//   cell
struct WalkMeta {
  int32_t src[4], push[kWalkPush], cell;
};
static_assert(sizeof(WalkMeta) == 32, "copied in 16-byte units");

// per batch: first position, positions, its mailbox barrier (-1: no new slot) and the slots that fill it
struct WalkBatch {
  int32_t first, n, bar, slots;
};
static_assert(sizeof(WalkBatch) == 16, "read as one vector");

struct WalkSchedule {
  int K = 1, parts = 1, ns = 2;  // ns: neighbour slots per record (2..4)
  int mail = 0, bars = 0;        // largest mailbox, most mailbox barriers of a block
  int maxBatches = 0;                      // of one block
  double time = 0;                         // estimated length of the walk in batches
  std::vector<int32_t> cells;              // [N] schedule order: part, run, level, cell
  std::vector<WalkMeta> meta;              // [N]
  std::vector<int32_t> nbF, nbJ;           // [N][4] per face slot: its face (cellFace code) and the neighbour that enters
                                           // this sweep (-1: none; kWalkGhost - j: in another part)
  std::vector<int32_t> blockBatch;         // [parts * K + 1] first batch of every block
  std::vector<WalkBatch> batches;
};
constexpr int32_t kWalkGhost = -2;

// the length of the walk in batches with one block per part; levels[p]: the levels of part p
inline double walk_length_one(int64_t N, int parts, const std::vector<int32_t>& part, const std::vector<int32_t>& level,
                              const std::vector<int32_t>& levels) {
  std::vector<int64_t> first(parts + 1, 0);
  for (int p = 0; p < parts; p++) first[p + 1] = first[p] + levels[p];
  std::vector<int32_t> width(first[parts], 0);
  for (int64_t i = 0; i < N; i++) width[first[part[i]] + level[i]]++;
  int64_t most = 0;
  for (int p = 0; p < parts; p++) {
    int64_t n = 0;
    for (int64_t l = first[p]; l < first[p + 1]; l++) n += (width[l] + kWalkW - 1) / kWalkW;
    most = std::max(most, n);
  }
  return (double)most;
}

// slotF / slotJ [N][4]: a cell's faces and the cells across (-1: none); pos: scan position; level: the
// cell's dependency level in this sweep.  False if the mailboxes of this K would need more than maxMail
// slots or a cell more than kWalkPush mailboxes; K = 1 always works.
inline bool build_walk(int64_t N, int parts, const std::vector<int32_t>& part, const std::vector<int32_t>& order,
                       const std::vector<int32_t>& pos, const std::vector<int32_t>& level, const std::vector<int32_t>& slotF,
                       const std::vector<int32_t>& slotJ, bool forward, int K, int maxMail, double hop, WalkSchedule& w) {
  w = WalkSchedule();
  w.K = K;
  w.parts = parts;
  const int nblk = parts * K;
  // runs: consecutive scan positions of a part
  std::vector<int64_t> count(parts, 0), seen(parts, 0);
  for (int64_t i = 0; i < N; i++) count[part[i]]++;
  std::vector<int32_t> blk(N);
  for (int64_t s = 0; s < N; s++) {
    const int32_t i = order[s], p = part[i];
    blk[i] = p * K + (int32_t)(seen[p]++ * K / count[p]);
  }
  // schedule order: block, level, cell
  int nlev = 0;
  for (int64_t i = 0; i < N; i++) nlev = std::max(nlev, level[i] + 1);
  std::vector<int64_t> at(nlev + 1, 0);
  for (int64_t i = 0; i < N; i++) at[level[i] + 1]++;
  for (int l = 0; l < nlev; l++) at[l + 1] += at[l];
  std::vector<int32_t> byLevel(N);
  for (int64_t i = 0; i < N; i++) byLevel[at[level[i]]++] = (int32_t)i;
  std::vector<int64_t> start(nblk + 1, 0), fill;
  for (int64_t i = 0; i < N; i++) start[blk[i] + 1]++;
  for (int b = 0; b < nblk; b++) start[b + 1] += start[b];
  fill.assign(start.begin(), start.end() - 1);
  w.cells.resize(N);
  for (int64_t t = 0; t < N; t++) w.cells[fill[blk[byLevel[t]]]++] = byLevel[t];
  std::vector<int32_t> posn(N), batchOf(N);
  w.blockBatch.assign(nblk + 1, 0);
  for (int b = 0; b < nblk; b++) {
    w.blockBatch[b] = (int32_t)w.batches.size();
    for (int64_t t = start[b]; t < start[b + 1]; t++) {
      const int32_t i = w.cells[t];
      if (t == start[b] || w.batches.back().n == kWalkW || level[i] != level[w.cells[t - 1]])
        w.batches.push_back(WalkBatch{(int32_t)t, 0, -1, 0});
      w.batches.back().n++;
      posn[i] = (int32_t)t;
      batchOf[i] = (int32_t)w.batches.size() - 1;
    }
    w.maxBatches = std::max<int>(w.maxBatches, (int)w.batches.size() - w.blockBatch[b]);
  }
  w.blockBatch[nblk] = (int32_t)w.batches.size();
  // neighbours
  w.meta.resize(N);
  w.nbF.assign(4 * N, -1);
  w.nbJ.assign(4 * N, -1);
  std::vector<int32_t> mail(nblk, 0), bars(nblk, 0);
  for (int64_t t = 0; t < N; t++) {
    for (int q = 0; q < 4; q++) w.meta[t].src[q] = 32 * kWalkZero;
    for (int q = 0; q < kWalkPush; q++) w.meta[t].push[q] = -1;
    w.meta[t].cell = w.cells[t];
  }
  for (int64_t t = 0; t < N; t++) {
    const int32_t i = w.cells[t], b = blk[i];
    int nu = 0;
    for (int k = 0; k < 4; k++) {
      const int32_t j = slotJ[4 * (int64_t)i + k];
      w.nbF[4 * t + k] = slotF[4 * (int64_t)i + k];
      if (j < 0) continue;
      if (part[j] != part[i]) {  // a ghost enters the backward sweep with its increment after the forward one
        if (!forward) w.nbJ[4 * t + k] = kWalkGhost - j;
        continue;
      }
      if (forward ? pos[j] >= pos[i] : pos[j] <= pos[i]) continue;
      w.nbJ[4 * t + k] = j;
      int32_t& src = w.meta[t].src[nu++];
      const int64_t pj = posn[j];
      if (blk[j] == b) {
        const int64_t end = (int64_t)w.batches[batchOf[i]].first + w.batches[batchOf[i]].n;
        src = pj + kWalkRing >= end ? (int32_t)((pj - start[b]) & (kWalkRing - 1)) * 32 : -(j + 1);
        continue;
      }
      int32_t* push = w.meta[pj].push;
      int q = 0;
      while (q < kWalkPush && push[q] >= 0 && (push[q] >> (2 * kWalkSlotBits)) != b % K) q++;
      if (q == kWalkPush) return false;
      if (push[q] < 0) {
        WalkBatch& x = w.batches[batchOf[i]];
        if (mail[b] >= std::min(maxMail, kWalkMaxMail)) return false;
        if (x.bar < 0) x.bar = bars[b]++;
        x.slots++;
        push[q] = walk_push(b % K, x.bar, mail[b]++);
      }
      src = (kWalkZero + 1 + (push[q] & kWalkMaxMail)) * 32;
    }
    w.ns = std::max(w.ns, nu);
  }
  w.mail = *std::max_element(mail.begin(), mail.end());
  w.bars = *std::max_element(bars.begin(), bars.end());
  // length of the walk: a batch takes 1, a value from another block `hop` more
  std::vector<double> done(w.batches.size(), 0.0);
  for (int p = 0; p < parts; p++)
    for (int c = 0; c < K; c++) {
      const int b = p * K + (forward ? c : K - 1 - c);
      double now = 0;
      for (int32_t x = w.blockBatch[b]; x < w.blockBatch[b + 1]; x++) {
        if (w.batches[x].bar >= 0)
          for (int64_t t = w.batches[x].first; t < w.batches[x].first + w.batches[x].n; t++)
            for (int k = 0; k < 4; k++) {
              const int32_t j = w.nbJ[4 * t + k];
              if (j >= 0 && blk[j] != b) now = std::max(now, done[batchOf[j]] + hop);
            }
        done[x] = ++now;
      }
      w.time = std::max(w.time, now);
    }
  return true;
}

}  // namespace dg
