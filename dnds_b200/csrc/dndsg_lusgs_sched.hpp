// dndsg_lusgs_sched.hpp -- host side of the scan-order LU-SGS sweep: which thread block walks which cells
// in which order, and where every neighbour's increment is when a cell needs it.  Plain C++, so that the
// schedule can be checked on the CPU.
//
// A sweep in scan order is a chain of dependency levels (a cell's level is one more than the largest
// level of its earlier neighbours).  Each part (the reference's rank) is cut into K runs of consecutive
// scan positions or of consecutive cells, one thread block per run, the K blocks of a part being one
// thread-block cluster.  A block walks its own cells level by level in batches of at most kWalkW cells (kWalkWide
// in parts of one block with wide levels), a block barrier between batches.  Every block takes its levels in order and
// a cell needs lower levels only, so the blocks never wait on one another in a circle.  A neighbour's increment is
// read from
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
constexpr int kWalkWide = 64;   // two cells per lane
constexpr double kWalkWideCost = 1.3;  // a wide batch (0.24-0.26 us, quads in natural order) in batches of kWalkW (0.19-0.2 us)
constexpr int kWalkRing = 256;  // positions in the ring (a power of two)
constexpr int kWalkMaxK = 16;   // blocks per part (one cluster)
constexpr int kWalkZero = kWalkRing;
constexpr int kWalkPush = 3;    // mailboxes that one cell's increment can go to
constexpr int kWalkSlotBits = 13, kWalkMaxMail = (1 << kWalkSlotBits) - 1;
// a mailbox and its barrier as one non-negative number: block of the part, barrier, slot
inline int32_t walk_push(int block, int bar, int slot) { return (block << (2 * kWalkSlotBits)) | (bar << kWalkSlotBits) | slot; }

// The walk's shared memory.  A record holds a position's matrix rows (dndsg_lusgs.cuh), x0[4] and its WalkMeta
constexpr int walk_rec_bytes(int ns) { return ns * 128 + 64; }   // 64 mod 128: 16-byte loads of a quarter warp (two positions)
                                                                 // meet no bank twice
constexpr int walk_rec5_bytes(int ns) { return ns * 32 + 16; }   // U5: rows, x0, padding (an odd number of 16-byte units)
constexpr int walk_stages(int width) { return width == kWalkW ? 6 : 4; }             // batches of records in flight
constexpr int kWalkCopy = 2;                                                         // copying warps
constexpr int walk_rows(bool sa) { return 4 * kWalkW + (sa ? 32 : 0); }              // threads that compute a batch: rows, U5
// two sets, the copying warps and the mailbox warp (a wide walk has no mailbox)
constexpr int walk_threads(bool sa, int width) { return 2 * walk_rows(sa) + 32 * kWalkCopy + (width == kWalkW ? 32 : 0); }
// the stages' barriers, the mailbox barriers, values, U5 values, the stages' records
constexpr size_t walk_smem(int ns, bool sa, int width, int mail, int bars) {
  return (((size_t)walk_stages(width) * 16 + (size_t)bars * 8 + 31) & ~(size_t)31) + (size_t)(kWalkZero + 1 + mail) * 32 +
         (sa ? ((size_t)(kWalkZero + 1 + mail) * 8 + 15) & ~(size_t)15 : 0) +
         (size_t)walk_stages(width) * width * (walk_rec_bytes(ns) + (sa ? walk_rec5_bytes(ns) : 0));
}
constexpr size_t kWalkSmemMax = 227 * 1024;
static_assert(walk_smem(4, true, kWalkWide, 0, 0) <= kWalkSmemMax && walk_smem(4, true, kWalkW, 0, 0) <= kWalkSmemMax, "one block fits");
// no more mailbox slots than this fit (walk_smem of the schedule itself decides)
constexpr int walk_max_mail(int ns, bool sa) { return (int)((kWalkSmemMax - walk_smem(ns, sa, kWalkW, 0, 0)) / (sa ? 40 : 32)); }

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
  int width = kWalkW;            // most cells of a batch
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
                              const std::vector<int32_t>& levels, int batch = kWalkW) {
  std::vector<int64_t> first(parts + 1, 0);
  for (int p = 0; p < parts; p++) first[p + 1] = first[p] + levels[p];
  std::vector<int32_t> width(first[parts], 0);
  for (int64_t i = 0; i < N; i++) width[first[part[i]] + level[i]]++;
  int64_t most = 0;
  for (int p = 0; p < parts; p++) {
    int64_t n = 0;
    for (int64_t l = first[p]; l < first[p + 1]; l++) n += (width[l] + batch - 1) / batch;
    most = std::max(most, n);
  }
  return (double)most;
}

// slotF / slotJ [N][4]: a cell's faces and the cells across (-1: none); pos: scan position; level: the
// cell's dependency level in this sweep.  False if the mailboxes of this K would need more than maxMail
// slots or a cell more than kWalkPush mailboxes; K = 1 always works.  width: cells per batch (kWalkWide: K = 1);
// byCell: runs of consecutive cells instead of scan positions.
inline bool build_walk(int64_t N, int parts, const std::vector<int32_t>& part, const std::vector<int32_t>& order,
                       const std::vector<int32_t>& pos, const std::vector<int32_t>& level, const std::vector<int32_t>& slotF,
                       const std::vector<int32_t>& slotJ, bool forward, int K, int maxMail, double hop, WalkSchedule& w,
                       int width = kWalkW, bool byCell = false) {
  w = WalkSchedule();
  w.K = K;
  w.parts = parts;
  w.width = width;
  const int nblk = parts * K;
  // runs: consecutive scan positions, or cells, of a part
  std::vector<int64_t> count(parts, 0), seen(parts, 0);
  for (int64_t i = 0; i < N; i++) count[part[i]]++;
  std::vector<int32_t> blk(N);
  for (int64_t s = 0; s < N; s++) {
    const int32_t i = byCell ? (int32_t)s : order[s], p = part[i];
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
      if (t == start[b] || w.batches.back().n == width || level[i] != level[w.cells[t - 1]])
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
  if (K == 1) {
    w.time = w.maxBatches;
    return true;
  }
  std::vector<double> done(w.batches.size(), 0.0), now(nblk, 0.0);
  std::vector<int32_t> next(w.blockBatch.begin(), w.blockBatch.end() - 1);
  for (int l = 0; l < nlev; l++)
    for (int b = 0; b < nblk; b++)
      for (; next[b] < w.blockBatch[b + 1] && level[w.cells[w.batches[next[b]].first]] == l; next[b]++) {
        const WalkBatch& x = w.batches[next[b]];
        if (x.bar >= 0)
          for (int64_t t = x.first; t < x.first + x.n; t++)
            for (int k = 0; k < 4; k++) {
              const int32_t j = w.nbJ[4 * t + k];
              if (j >= 0 && blk[j] != b) now[b] = std::max(now[b], done[batchOf[j]] + hop);
            }
        done[next[b]] = ++now[b];
      }
  w.time = *std::max_element(now.begin(), now.end());
  return true;
}

// The schedules of both sweeps.  A part is walked by a cluster of blocks, one per 8 cells of a mean level, where the
// lengths of the walks make that shorter than one block; sweeps of quads in natural order, us (lengths):
//                              one block     one block, wide   cluster of 16 or 8
//   512 x 128, 103 a level     462 (2172)      315 (1495)         157 (684)
//   1000 x 70, 65 a level      620 (3015)      565 (2613)         250 (2119)
//   256 x 64, 51 a level       127 (574)        91 (415)           81 (340)
// The blocks have runs of consecutive scan positions, or of cells where those of the scan order do not fit (an order that
// jumps about the mesh: its neighbours are in other runs), and there are half as many where those do not either: when
// the walk does not get shorter by them, the mailboxes do not fit the shared memory, or the device (fits(ns, K, mail,
// bars)) does not take such a cluster.
template <class Fits>
inline void choose_walks(int64_t N, int parts, const std::vector<int32_t>& part, const std::vector<int32_t>& order,
                         const std::vector<int32_t>& pos, const std::vector<int32_t>& lf, const std::vector<int32_t>& nlf,
                         const std::vector<int32_t>& lb, const std::vector<int32_t>& nlb, const std::vector<int32_t>& slotF,
                         const std::vector<int32_t>& slotJ, bool sa, int sms, double hop, Fits&& fits, WalkSchedule& fwd,
                         WalkSchedule& bwd) {
  const int levels = *std::max_element(nlf.begin(), nlf.end()) + *std::max_element(nlb.begin(), nlb.end());
  auto length = [&](int width) {
    return walk_length_one(N, parts, part, lf, nlf, width) + walk_length_one(N, parts, part, lb, nlb, width);
  };
  const double one = length(kWalkW), wide = kWalkWideCost * length(kWalkWide);
  int K = 1;
  if (one > 1.05 * levels) {
    K = 2;
    while (K < kWalkMaxK && K * 8.0 < 2.0 * N / levels / parts) K *= 2;
    while (K > 1 && (int64_t)parts * K > sms) K /= 2;
  }
  bool natural = true, reverse = true;  // the runs are those of the cells anyway
  for (int64_t s = 0; s < N && (natural || reverse); s++) {
    natural = natural && order[s] == s;
    reverse = reverse && order[s] == N - 1 - s;
  }
  for (; K > 1; K /= 2)
    for (int byCell = 0; byCell < (natural || reverse ? 1 : 2); byCell++) {
      auto build = [&](bool forward, WalkSchedule& w) {
        return build_walk(N, parts, part, order, pos, forward ? lf : lb, slotF, slotJ, forward, K, walk_max_mail(2, sa), hop, w,
                          kWalkW, byCell) &&
               walk_smem(w.ns, sa, kWalkW, w.mail, w.bars) <= kWalkSmemMax && fits(w.ns, K, w.mail, w.bars);
      };
      if (build(true, fwd) && build(false, bwd) && fwd.time + bwd.time < 0.95 * std::min(one, wide)) return;
    }
  const int width = wide < one ? kWalkWide : kWalkW;
  build_walk(N, parts, part, order, pos, lf, slotF, slotJ, true, 1, 0, hop, fwd, width);
  build_walk(N, parts, part, order, pos, lb, slotF, slotJ, false, 1, 0, hop, bwd, width);
}

}  // namespace dg
