// Host plan of the block ILU sweeps (k_ilu_sweep_cluster in ilu.cuh): which
// rows are solved together, by which thread block, and where each solved
// value goes.
//
// The rows of a triangle form a dependency graph; any topological order
// gives every row the same arithmetic.  Plain levels (each row as early as
// its dependencies allow) are uneven -- 74,528 rows: 492 levels of 1 to 689
// rows -- and a wide level is one that the thread blocks of a cluster would
// walk in several rounds.  Here the rows are list-scheduled: per level at
// most cluster * kSweepRows rows, the most urgent first (longest chain of
// rows still to come).  That keeps the number of levels (492) and caps their
// width at what one round solves.  Every level starts at a multiple of 32
// positions; positions past its rows are padding.
//
// Each dependency has a slot of its own in the shared memory of the block
// that solves the row, given out for the levels from the solve of the value
// to its use; the block that solves the value writes it there and counts it
// on that block's barrier of level min(use, solve + kSweepNear).  Blocks may
// be up to kSweepSkew levels apart, so a slot is given out again kSweepSkew
// levels after its use at the earliest, and kSweepBars level barriers exist
// at once.
//
// Record of a position (kSweepRec int32):
//   [0]     row, -1 padding
//   [1]     number of dependencies
//   [2..3]  their operand slots, slot order, 16 bits each
//   [4..7]  where the solved value goes, -1 none:
//           block << 16 | barrier << 12 | operand slot
//   [8]     the row's backward position
//   [9]     matrix slot of each dependency, 8 bits each
// Entry of a level and block (info, 4 int32): first chunk (the others follow
// `cluster` apart), chunks, bit set of the chunks with more than two
// dependencies in a row, bytes its barrier of the level waits for.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#if defined(__CUDACC__)
#define O2F_PLAN_FN __host__ __device__ __forceinline__
#else
#define O2F_PLAN_FN inline
#endif

namespace o2f {

constexpr int kSweepChunks = 2;                // 32-row chunks of a level per thread block
constexpr int kSweepRows = 32 * kSweepChunks;  // rows of a level per thread block
constexpr int kSweepRec = 12;                  // int32 per record
constexpr int kSweepSlots = 2048;              // operand slots per block
constexpr int kSweepBars = 16;                 // level barriers per block
constexpr int kSweepNear = 8;                  // levels ahead that a value can be counted on
constexpr int kSweepSkew = 8;                  // levels that blocks can be apart
constexpr int kSweepMaxCluster = 8;            // portable cluster size
static_assert(kSweepNear + kSweepSkew <= kSweepBars, "a barrier's phases would overlap");
static_assert(kSweepSlots <= 4096 && kSweepBars <= 16, "fields of a target");

struct SweepPlan {
  int cluster = 0;                    // 0: no plan (a block's operand slots ran out)
  int nlev[2] = {0, 0};               // forward, backward
  int64_t chunks[2] = {0, 0};
  std::vector<int32_t> info[2];       // [nlev * cluster * 4]
  std::vector<int32_t> rec[2];        // [32 * chunks * kSweepRec]
  std::vector<int32_t> pos[2];        // [n] position of each row
};

// Place of element el of the 4x4 block of row q of a chunk inside the 512
// doubles of the chunk's blocks: the two halves of a block row, then (row,
// component), so that a warp's four lanes per row read 16 consecutive bytes
// each, all 32 lanes 512.
O2F_PLAN_FN int sweep_pack_place(int q, int el) {
  return ((el >> 1) & 1) * 256 + (q * 4 + (el >> 2)) * 2 + (el & 1);
}

// Thread blocks per cluster: enough for the mean level in one round with a
// quarter to spare, so that the cap costs no levels.
inline int sweep_cluster_size(int64_t n, int nlev) {
  int c = 1;
  while (c < kSweepMaxCluster && (int64_t)c * kSweepRows * nlev * 4 < n * 5) c *= 2;
  return c;
}

// nbr: [4 * n] neighbours, slot-major, -1 none; pos: elimination position of
// each row; order: the rows by position.  cluster <= 0: chosen by size.
inline SweepPlan make_sweep_plan(int64_t n, const std::vector<int32_t>& nbr, const std::vector<int32_t>& pos,
                                 const std::vector<int32_t>& order, int cluster = 0) {
  SweepPlan pl;
  auto before = [&](int dir, int32_t a, int32_t b) { return dir == 0 ? pos[a] < pos[b] : pos[a] > pos[b]; };
  // Forward levels.  Latest level of each row: from the ends of the chains back.
  std::vector<int32_t> late(n, 0), level[2];
  int depth = 0;
  for (int64_t i = n - 1; i >= 0; --i) {
    const int32_t c = order[i];
    int32_t h = 0;
    for (int k = 0; k < 4; ++k) {
      const int32_t o = nbr[k * n + c];
      if (o >= 0 && before(0, c, o)) h = std::max(h, late[o] + 1);
    }
    late[c] = h;
    depth = std::max(depth, h + 1);
  }
  for (auto& h : late) h = depth - 1 - h;
  const int C = cluster > 0 ? cluster : sweep_cluster_size(n, std::max(1, depth));
  const int cap = C * kSweepRows;
  level[0].assign(n, -1);
  // ready rows by urgency: stacks linked through `next`, one per latest level
  std::vector<int32_t> head(depth + 1, -1), next(n, -1);
  std::vector<uint8_t> left(n, 0);
  int top = depth, nlev = 0;
  auto ready = [&](int32_t c) {
    next[c] = head[late[c]];
    head[late[c]] = c;
    top = std::min(top, (int)late[c]);
  };
  for (int64_t i = n - 1; i >= 0; --i) {
    const int32_t c = order[i];
    for (int k = 0; k < 4; ++k) {
      const int32_t o = nbr[k * n + c];
      left[c] += o >= 0 && before(0, o, c);
    }
    if (left[c] == 0) ready(c);
  }
  std::vector<int32_t> take;
  std::vector<int64_t> width;
  for (int64_t done = 0; done < n; done += (int64_t)take.size()) {
    // the rows that cannot wait, and of the others an even share: a row
    // solved long before it is needed holds operand slots
    const int64_t levels_left = std::max<int64_t>(1, depth - nlev);
    const int share = (int)std::min<int64_t>(cap, (n - done + levels_left - 1) / levels_left);
    take.clear();
    while ((int)take.size() < cap && top < depth) {
      const int32_t c = head[top];
      if (c < 0) {
        ++top;
        continue;
      }
      if (top > nlev && (int)take.size() >= share) break;
      head[top] = next[c];
      take.push_back(c);
    }
    if (take.empty()) return SweepPlan{};  // a cycle: cannot happen for an elimination order
    for (int32_t c : take) level[0][c] = nlev;
    for (int32_t c : take)
      for (int k = 0; k < 4; ++k) {
        const int32_t o = nbr[k * n + c];
        if (o >= 0 && before(0, c, o) && --left[o] == 0) ready(o);
      }
    width.push_back((int64_t)take.size());
    ++nlev;
  }
  // The backward triangle's dependencies are the forward ones reversed, and
  // so are its levels (scheduled by themselves they need up to three times
  // the operand slots).
  level[1].resize(n);
  for (int64_t c = 0; c < n; ++c) level[1][c] = nlev - 1 - level[0][c];
  std::vector<int32_t> off[2];
  for (int dir = 0; dir < 2; ++dir) {
    pl.nlev[dir] = nlev;
    off[dir].assign(1, 0);
    std::vector<int32_t> fill(nlev);
    for (int l = 0; l < nlev; ++l) {
      fill[l] = 32 * off[dir].back();
      off[dir].push_back(off[dir].back() + (int32_t)((width[dir == 0 ? l : nlev - 1 - l] + 31) / 32));
    }
    // rows of a level in elimination order: their dependencies are close too
    pl.pos[dir].assign(n, -1);
    for (int64_t i = 0; i < n; ++i) pl.pos[dir][order[i]] = fill[level[dir][order[i]]]++;
    pl.chunks[dir] = off[dir].back();
  }
  for (int dir = 0; dir < 2; ++dir) {
    std::vector<int32_t>&rec = pl.rec[dir], &info = pl.info[dir];
    rec.assign((size_t)pl.chunks[dir] * 32 * kSweepRec, -1);
    info.assign((size_t)nlev * C * 4, 0);
    for (int l = 0; l < nlev; ++l)
      for (int b = 0; b < C; ++b) {
        int32_t* in = info.data() + ((size_t)l * C + b) * 4;
        in[0] = off[dir][l] + b;
        for (int k = in[0]; k < off[dir][l + 1]; k += C) ++in[1];
      }
    for (int64_t c = 0; c < n; ++c) {
      int32_t* r = rec.data() + (size_t)pl.pos[dir][c] * kSweepRec;
      r[0] = (int32_t)c;
      r[1] = 0;
      r[8] = pl.pos[1][c];
    }
    // operand slots of each block: free ones, and those that become free at a level
    std::vector<std::vector<int32_t>> free_slots(C);
    std::vector<std::vector<std::pair<int32_t, int32_t>>> back(nlev + kSweepSkew + 1);
    for (auto& f : free_slots)
      for (int s = kSweepSlots; s-- > 0;) f.push_back(s);
    for (int l = 0; l < nlev; ++l) {
      for (auto& [b, s] : back[l]) free_slots[b].push_back(s);
      for (int64_t p = (int64_t)off[dir][l] * 32; p < (int64_t)off[dir][l + 1] * 32; ++p) {
        int32_t* r = rec.data() + (size_t)p * kSweepRec;
        const int32_t c = r[0];
        if (c < 0) continue;
        int t = 4;
        for (int k = 0; k < 4; ++k) {  // the rows that need c's value
          const int32_t o = nbr[k * n + c];
          if (o < 0 || !before(dir, c, o)) continue;
          const int32_t po = pl.pos[dir][o], lo = level[dir][o], at = (po >> 5) - off[dir][lo], b = at % C;
          if (free_slots[b].empty()) return SweepPlan{};
          const int32_t s = free_slots[b].back();
          free_slots[b].pop_back();
          back[lo + kSweepSkew].emplace_back(b, s);
          const int32_t bar = std::min(lo, l + kSweepNear);
          info[((size_t)bar * C + b) * 4 + 3] += 32;
          r[t++] = (b << 16) | ((bar % kSweepBars) << 12) | s;
          // which of o's dependencies this is (cells can share two edges)
          int same = 0, d = 0;
          for (int q = 0; q < k; ++q) same += nbr[q * n + c] == o;
          for (int q = 0;; ++q) {
            const int32_t x = nbr[q * n + o];
            if (x == c && same-- == 0) break;
            d += x >= 0 && before(dir, x, o);
          }
          int32_t& w = rec[(size_t)po * kSweepRec + 2 + d / 2];
          w = d % 2 == 0 ? (int32_t)(((uint32_t)w & 0xffff0000u) | (uint32_t)s)
                         : (int32_t)(((uint32_t)w & 0xffffu) | ((uint32_t)s << 16));
        }
        uint32_t slots = 0xffffffffu;
        for (int k = 0; k < 4; ++k) {
          const int32_t o = nbr[k * n + c];
          if (o < 0 || !before(dir, o, c)) continue;
          slots = (slots & ~(0xffu << (8 * r[1]))) | ((uint32_t)k << (8 * r[1]));
          ++r[1];
        }
        r[9] = (int32_t)slots;
        if (r[1] > 2) {
          const int32_t at = (int32_t)(p >> 5) - off[dir][l];
          info[((size_t)l * C + at % C) * 4 + 2] |= 1 << (at / C);
        }
      }
    }
  }
  pl.cluster = C;
  return pl;
}

}  // namespace o2f
