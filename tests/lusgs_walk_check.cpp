// Walks LU-SGS schedules (dnds_b200/csrc/dndsg_lusgs_sched.hpp) on the host, the blocks of a part in random
// turns, and checks that every increment a cell reads is the one of the neighbour the sequential sweep
// reads there.  Usage: lusgs_walk_check nx ny tri parts order K seed; prints the blocks' batches.  K = -1: one
// block, wide batches; K < -1: runs of cells instead of scan positions; K = 0: the blocks per part and the batch width that choose_walks takes, without and with U5.
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>
#include <set>

#include "dndsg_lusgs_sched.hpp"
using namespace dg;

#define REQUIRE(x) do { if (!(x)) { std::printf("failed: %s (line %d)\n", #x, __LINE__); return 1; } } while (0)

int main(int, char** a) {
  const int nx = std::abs(std::atoi(a[1])), ny = std::atoi(a[2]), tri = std::atoi(a[3]), P = std::atoi(a[4]), order = std::atoi(a[5]),
            K0 = std::atoi(a[6]), K = std::abs(K0), width = K0 == -1 ? kWalkWide : kWalkW, maxMail = 100000;
  std::mt19937 rng(std::atoi(a[7]));
  // a grid of quads, or each split in two, periodic in x (nx < 0: not); every cell's neighbours across its faces
  const bool periodic = std::atoi(a[1]) > 0;
  const int64_t N = (int64_t)nx * ny * (tri ? 2 : 1);
  std::vector<int32_t> slotF(4 * N, -1), slotJ(4 * N, -1), fill(N, 0);
  int faces = 0;
  auto join = [&](int64_t p, int64_t q) {
    slotF[4 * p + fill[p]] = faces;
    slotJ[4 * p + fill[p]++] = (int32_t)q;
    slotF[4 * q + fill[q]] = ~faces++;
    slotJ[4 * q + fill[q]++] = (int32_t)p;
  };
  for (int64_t j = 0; j < ny; j++)
    for (int64_t i = 0; i < nx; i++) {
      const int64_t c = i * ny + j, r = periodic || i + 1 < nx ? (i + 1) % nx * ny + j : c;
      if (tri) {
        join(2 * c, 2 * c + 1);
        if (r != c) join(2 * c + 1, 2 * r);
        if (j + 1 < ny) join(2 * c + 1, 2 * (c + 1));
      } else {
        if (r != c) join(c, r);
        if (j + 1 < ny) join(c, c + 1);
      }
    }
  std::vector<int32_t> scan(N), pos(N), part(N);
  std::iota(scan.begin(), scan.end(), 0);
  if (order == 1) std::reverse(scan.begin(), scan.end());
  if (order >= 2) std::shuffle(scan.begin(), scan.end(), rng);
  if (order == 4) {  // lines of the slower direction, even ones first
    int64_t s = 0;
    for (int odd = 0; odd < 2; odd++)
      for (int64_t c = 0; c < N; c++)
        if (c / (N / nx) % 2 == odd) scan[s++] = (int32_t)c;
  }
  for (int64_t s = 0; s < N; s++) pos[scan[s]] = (int32_t)s;
  for (int64_t i = 0; i < N; i++) part[i] = order == 2 ? (int32_t)(rng() % P) : (int32_t)(i * P / N);
  auto levels = [&](bool forward) {
    std::vector<int32_t> level(N, 0);
    for (int64_t x = 0; x < N; x++) {
      const int32_t i = scan[forward ? x : N - 1 - x];
      for (int k = 0; k < 4; k++) {
        const int32_t j = slotJ[4 * (int64_t)i + k];
        if (j >= 0 && part[j] == part[i] && (forward ? pos[j] < pos[i] : pos[j] > pos[i])) level[i] = std::max(level[i], level[j] + 1);
      }
    }
    return level;
  };
  if (K == 0) {
    const std::vector<int32_t> lf = levels(true), lb = levels(false);
    std::vector<int32_t> nlf(P, 0), nlb(P, 0);
    for (int64_t i = 0; i < N; i++) {
      nlf[part[i]] = std::max(nlf[part[i]], lf[i] + 1);
      nlb[part[i]] = std::max(nlb[part[i]], lb[i] + 1);
    }
    for (int sa = 0; sa < 2; sa++) {
      WalkSchedule f, b;
      choose_walks(N, P, part, scan, pos, lf, nlf, lb, nlb, slotF, slotJ, sa, 148, 3.0, [](int, int, int, int) { return true; }, f, b);
      REQUIRE(f.K == b.K && f.width == b.width && (f.width == kWalkW || f.K == 1));
      for (const WalkSchedule* w : {&f, &b}) REQUIRE(walk_smem(w->ns, sa, w->width, w->mail, w->bars) <= kWalkSmemMax);
      std::printf("%dx%d ", f.K, f.width);
    }
    return 0;
  }
  int built = 0;
  for (int forward = 1; forward >= 0; forward--) {
    const std::vector<int32_t> level = levels(forward);
    WalkSchedule w;
    if (!build_walk(N, P, part, scan, pos, level, slotF, slotJ, forward, K, maxMail, 3.0, w, width, K0 < -1)) {
      REQUIRE(K > 1);
      continue;
    }
    built++;
    const int nblk = P * K;
    REQUIRE((int64_t)w.cells.size() == N && (int)w.blockBatch.size() == nblk + 1 && w.mail <= maxMail);
    REQUIRE(std::set<int32_t>(w.cells.begin(), w.cells.end()).size() == (size_t)N);
    // per block: the shared slots hold the cell whose increment they carry; `global` the cells stored
    std::vector<std::vector<int32_t>> slots(nblk, std::vector<int32_t>(kWalkZero + 1 + w.mail, -1));
    std::vector<int32_t> done(nblk, 0), stored(N, -1), batchOf(N, -1);  // batchOf: the batch that stored a cell
    std::vector<std::vector<int32_t>> filled(nblk, std::vector<int32_t>(w.bars, 0));  // slots filled per mailbox barrier
    int64_t left = (int64_t)w.batches.size();
    REQUIRE(w.blockBatch[nblk] == left);
    int idle = 0;
    while (left > 0) {
      REQUIRE(idle < 100000);  // no block can go on
      const int b = (int)(rng() % nblk), first = b / K * K;
      const int32_t x = w.blockBatch[b] + done[b];
      idle++;
      if (x == w.blockBatch[b + 1]) continue;
      const WalkBatch& bt = w.batches[x];
      REQUIRE(bt.bar < w.bars && (bt.bar >= 0) == (bt.slots > 0));
      const bool ready = bt.bar < 0 || filled[b][bt.bar] == bt.slots;
      if (!ready) continue;
      idle = 0;
      REQUIRE(bt.n >= 1 && bt.n <= width);
      REQUIRE(x + 1 == (int32_t)w.batches.size() ? bt.first + bt.n == N : bt.first + bt.n == w.batches[x + 1].first);
      const int32_t p0 = w.batches[w.blockBatch[b]].first;
      for (int32_t t = bt.first; t < bt.first + bt.n; t++) {
        const int32_t i = w.meta[t].cell;
        REQUIRE(i == w.cells[t] && part[i] == b / K);
        int nu = 0;
        for (int k = 0; k < 4; k++) {
          const int32_t j = slotJ[4 * (int64_t)i + k];
          const bool same = j >= 0 && part[j] == part[i], used = same && (forward ? pos[j] < pos[i] : pos[j] > pos[i]);
          REQUIRE(w.nbF[4 * (int64_t)t + k] == slotF[4 * (int64_t)i + k]);
          REQUIRE(w.nbJ[4 * (int64_t)t + k] == (used ? j : (j >= 0 && !same && !forward ? kWalkGhost - j : -1)));
          if (!used) continue;
          int32_t src = w.meta[t].src[nu++];
          REQUIRE(src < 0 || src % 32 == 0);
          if (src >= 0) src /= 32;
          // global memory: only the block's own cells, stored after their batch's barrier and so seen two further on
          if (src < 0) REQUIRE(-src - 1 == j && stored[j] == b && batchOf[j] + 2 <= x - 1);
          else {
            REQUIRE(src != kWalkZero && src < kWalkZero + 1 + w.mail);
            REQUIRE(slots[b][src] == j);
          }
        }
        REQUIRE(nu <= w.ns);
        for (int q = nu; q < 4; q++) REQUIRE(w.meta[t].src[q] == 32 * kWalkZero);
      }
      for (int32_t t = bt.first; t < bt.first + bt.n; t++) {  // a batch's reads are before its stores or beside them:
        const int32_t i = w.meta[t].cell;                      // check the slots it overwrites are not read in it
        const int32_t sl = (t - p0) & (kWalkRing - 1);
        for (int32_t u = bt.first; u < bt.first + bt.n; u++)
          for (int q = 0; q < 4; q++) REQUIRE(w.meta[u].src[q] != 32 * sl);
        stored[i] = b;
        batchOf[i] = x;
        for (int q = 0; q < kWalkPush && w.meta[t].push[q] >= 0; q++) {
          const int32_t x = w.meta[t].push[q];
          const int to = x >> (2 * kWalkSlotBits), bar = x >> kWalkSlotBits & kWalkMaxMail, m = x & kWalkMaxMail;
          REQUIRE(to < K && to != b - first && m < w.mail && bar < w.bars);
          REQUIRE(slots[first + to][kWalkZero + 1 + m] == -1);  // a mailbox slot is written once
          filled[first + to][bar]++;
          slots[first + to][kWalkZero + 1 + m] = i;
        }
      }
      for (int32_t t = bt.first; t < bt.first + bt.n; t++) slots[b][(t - p0) & (kWalkRing - 1)] = w.meta[t].cell;
      done[b]++;
      left--;
    }
    if (K == 1) {
      std::vector<int32_t> levels(P, 0);
      for (int64_t i = 0; i < N; i++) levels[part[i]] = std::max(levels[part[i]], level[i] + 1);
      REQUIRE(walk_length_one(N, P, part, level, levels, width) == w.time);
    }
    std::printf("%s: %d blocks, at most %d batches, length %.0f, %d slots, mail %d, barriers %d\n", forward ? "forward" : "backward", nblk, w.maxBatches,
                w.time, w.ns, w.mail, w.bars);
  }
  std::printf("ok %d\n", built);
  return 0;
}
