// Host check of the block ILU sweeps' plan (csrc/sweep_plan.hpp): walks each
// triangle level by level as k_ilu_sweep_cluster does, with a tag of the row
// as its value, and checks that every row is solved once, that every
// dependency's value is in its operand slot and counted on a barrier the row
// has waited for, that no slot is written again while a block may still read
// it, and that all indices stay inside the buffers; then runs the kernel's synchronisation with warps and values in
// random order.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "sweep_plan.hpp"

using namespace o2f;

#define CHECK(x)                                                            \
  do {                                                                      \
    if (!(x)) {                                                             \
      std::printf("FAILED %s (line %d)\n", #x, __LINE__);                   \
      std::exit(1);                                                         \
    }                                                                       \
  } while (0)

static void walk(const SweepPlan& pl, int dir, int64_t n, const std::vector<int32_t>& nbr,
                 const std::vector<int32_t>& pos) {
  const int C = pl.cluster, nlev = pl.nlev[dir];
  const auto &info = pl.info[dir], &rec = pl.rec[dir];
  CHECK(info.size() == (size_t)nlev * C * 4);
  CHECK(rec.size() == (size_t)pl.chunks[dir] * 32 * kSweepRec);
  std::vector<std::vector<int32_t>> op(C, std::vector<int32_t>(kSweepSlots, -1));
  // level of the last use of a slot's value; while it waits for it, nlev
  std::vector<std::vector<int>> used(C, std::vector<int>(kSweepSlots, -1000));
  std::vector<std::vector<int64_t>> bytes(nlev, std::vector<int64_t>(C, 0));  // counted on each level's barrier
  std::vector<char> done(n, 0), seen(pl.chunks[dir], 0);
  for (int l = 0; l < nlev; ++l) {
    std::vector<int32_t> solved;
    struct Push {
      int rank, bar, slot;
      int32_t row;
    };
    std::vector<Push> push;
    for (int b = 0; b < C; ++b) {
      const int32_t* in = info.data() + ((size_t)l * C + b) * 4;
      CHECK(in[1] >= 0 && in[1] <= kSweepChunks);
      // what the barrier of this level waits for has been sent by earlier levels
      CHECK(bytes[l][b] == in[3] && in[3] < (1 << 20));
      for (int j = 0; j < in[1]; ++j) {
        const int64_t k = in[0] + (int64_t)j * C;
        CHECK(k < pl.chunks[dir] && !seen[k]);
        seen[k] = 1;
        for (int q = 0; q < 32; ++q) {
          const int64_t p = k * 32 + q;
          const int32_t* r = rec.data() + (size_t)p * kSweepRec;
          const int32_t c = r[0];
          if (c < 0) continue;
          CHECK(c < n && pl.pos[dir][c] == p && !done[c]);
          CHECK(r[8] == pl.pos[1][c]);
          const int nd = r[1];
          CHECK(nd <= 2 || (in[2] >> j & 1));
          int d = 0;
          for (int s = 0; s < 4; ++s) {
            const int32_t o = nbr[s * n + c];
            if (o < 0 || !(dir == 0 ? pos[o] < pos[c] : pos[o] > pos[c])) continue;
            CHECK(d < nd && done[o]);
            CHECK((int)(((uint32_t)r[9] >> (8 * d)) & 0xff) == s);
            const int slot = ((uint32_t)r[2 + d / 2] >> (16 * (d % 2))) & 0xffff;
            CHECK(slot < kSweepSlots && op[b][slot] == o && used[b][slot] == nlev);
            used[b][slot] = l;
            ++d;
          }
          CHECK(d == nd);
          bool end = false;
          for (int t = 4; t < 8; ++t) {
            if (r[t] < 0) end = true;
            else {
              CHECK(!end);  // targets come first
              push.push_back({r[t] >> 16, r[t] >> 12 & 15, r[t] & 0xfff, c});
            }
          }
          solved.push_back(c);
        }
      }
    }
    for (int32_t c : solved) done[c] = 1;
    for (const Push& u : push) {
      CHECK(u.rank < C && u.slot < kSweepSlots);
      // no block can still read the slot's last value
      CHECK(used[u.rank][u.slot] <= l - kSweepSkew);
      used[u.rank][u.slot] = nlev;
      op[u.rank][u.slot] = u.row;
      int bar = l + 1;  // the level that counts it: the next with its barrier
      while (bar % kSweepBars != u.bar) ++bar;
      CHECK(bar <= l + kSweepNear && bar < nlev);
      bytes[bar][u.rank] += 32;
    }
  }
  for (int64_t c = 0; c < n; ++c) CHECK(done[c]);
  for (auto& f : used)
    for (int v : f) CHECK(v < nlev);  // every value was used
}

// The kernel's synchronisation with its warps and the delivery of values in
// random order: mbarriers (phase, pending arrivals, bytes), the cluster
// barrier every 4 levels, staging slots.  A wait passes as the hardware's
// parity test does; checked: a wait never passes early, a row reads the
// values it needs, nothing is left waiting for ever.
struct Bar {
  int count, pending, done = 0;  // phases completed
  int64_t tx = 0;
  explicit Bar(int c) : count(c), pending(c) {}
  void settle() {
    if (pending == 0 && tx == 0) ++done, pending = count;
  }
  void arrive(int64_t expect) {
    CHECK(pending > 0);
    tx += expect;
    --pending;
    settle();
  }
  void complete(int64_t b) {
    tx -= b;
    settle();
  }
  bool passes(int phase) const { return (done & 1) != (phase & 1); }  // parity of the running phase
};

static void simulate(const SweepPlan& pl, int dir, int64_t n, const std::vector<int32_t>& nbr,
                     const std::vector<int32_t>& pos, std::mt19937& rng) {
  constexpr int kRing = 4, kWarps = 4 * kSweepChunks;  // warps of a level; two sets of them take turns
  constexpr int kSolve = 2 * kWarps, kAll = kSolve + kRing + 1;
  const int C = pl.cluster, nlev = pl.nlev[dir];
  const auto &info = pl.info[dir], &rec = pl.rec[dir];
  auto in = [&](int l, int b, int f) { return info[((size_t)l * C + b) * 4 + f]; };
  struct Block {
    std::vector<Bar> op, full, empty;
    std::vector<int> staged;  // level staged in a slot
    std::vector<int32_t> slot;
    Block()
        : op(kSweepBars, Bar(1)), full(kRing, Bar(1)), empty(kRing, Bar(kWarps)),
          staged(kRing, -1), slot(kSweepSlots, -1) {}
  };
  std::vector<Block> blk(C);
  struct Flight {
    int rank, bar, slot;
    int32_t row;
    int level;
  };
  std::vector<Flight> flight;
  struct Actor {  // a warp: level (-1: prologue), step 0 cluster barrier, 1 wait and work, 2 load the next
    int level = -1, step = 0, arrivals = 0;  // level: the first of a solving warp's pair, a staging warp's four
  };
  std::vector<Actor> act(C * kAll);
  auto all_arrived = [&](int k) {
    for (auto& a : act)
      if (a.arrivals < k) return false;
    return true;
  };
  auto stage = [&](int b, int l) {
    if (l >= nlev) return;
    Bar& f = blk[b].full[l % kRing];
    CHECK(f.done == l / kRing);
    blk[b].staged[l % kRing] = l;
    f.arrive(0);
  };
  auto arm = [&](int b, int l) {
    if (l >= nlev) return;
    Bar& o = blk[b].op[l % kSweepBars];
    CHECK(o.done == l / kSweepBars);
    o.arrive(in(l, b, 3));
  };
  auto load = [&](Block& B, int l) {  // a warp takes its rows of a staged level into registers
    Bar& f = B.full[l % kRing];
    if (!f.passes(l / kRing)) return false;
    CHECK(f.done == l / kRing + 1);
    CHECK(B.staged[l % kRing] == l);
    B.empty[l % kRing].arrive(0);
    return true;
  };
  int64_t idle = 0;
  int finished = 0;
  while (finished < C * kAll) {
    CHECK(++idle < 2000000);  // nothing moves: a deadlock
    if (!flight.empty() && rng() % 3 == 0) {
      const size_t i = rng() % flight.size();
      const Flight f = flight[i];
      flight[i] = flight.back();
      flight.pop_back();
      CHECK(blk[f.rank].op[f.bar].done == f.level / kSweepBars);
      blk[f.rank].slot[f.slot] = f.row;
      blk[f.rank].op[f.bar].complete(32);
      idle = 0;
    }
    const int who = (int)(rng() % act.size()), b = who / kAll, w = who % kAll;
    Actor& a = act[who];
    Block& B = blk[b];
    if (a.level >= nlev) continue;
    if (a.level < 0) {  // prologue
      if (w >= kSolve && w < kSolve + kRing) stage(b, w - kSolve);
      if (w == kSolve + kRing)
        for (int l = 0; l < kSweepNear; ++l) arm(b, l);
      if (w < kSolve && w / kWarps < nlev && !load(B, w / kWarps)) continue;
      a.level = 0;
      idle = 0;
      continue;
    }
    const int l = a.level + (w < kSolve ? w / kWarps : w < kSolve + kRing ? w - kSolve : 0);
    if (a.step == 0) {
      if (a.level % (kSweepSkew / 2) == 0) {
        if (a.level > 0 && !all_arrived(a.level / (kSweepSkew / 2))) continue;
        ++a.arrivals;
      }
      a.step = 1;
    } else if (l >= nlev) {
      a.level = nlev;
      ++finished;
    } else if (a.step == 1) {
      if (w < kSolve) {
        Bar& o = B.op[l % kSweepBars];
        if (!o.passes(l / kSweepBars)) continue;
        CHECK(o.done == l / kSweepBars + 1);
        const int j = w / 4 % kSweepChunks;
        if (j < in(l, b, 1)) {
          const int64_t k = in(l, b, 0) + (int64_t)j * C;
          for (int q = w % 4 * 8; q < w % 4 * 8 + 8; ++q) {
            const int32_t* r = rec.data() + (size_t)(k * 32 + q) * kSweepRec;
            if (r[0] < 0) continue;
            int d = 0;
            for (int s = 0; s < 4; ++s) {
              const int32_t x = nbr[s * n + r[0]];
              if (x < 0 || !(dir == 0 ? pos[x] < pos[r[0]] : pos[x] > pos[r[0]])) continue;
              CHECK(B.slot[((uint32_t)r[2 + d / 2] >> (16 * (d % 2))) & 0xffff] == x);
              ++d;
            }
            for (int t = 4; t < 8 && r[t] >= 0; ++t) {
              int bar = l + 1;
              while (bar % kSweepBars != (r[t] >> 12 & 15)) ++bar;
              flight.push_back({r[t] >> 16, r[t] >> 12 & 15, r[t] & 0xfff, r[0], bar});
            }
          }
        }
      } else if (w < kSolve + kRing) {
        if (!B.empty[l % kRing].passes(l / kRing)) continue;
        CHECK(B.empty[l % kRing].done == l / kRing + 1);
        stage(b, l + kRing);
      } else {
        arm(b, l + kSweepNear);
      }
      a.step = 2;
    } else {
      if (w < kSolve && l + 2 < nlev && !load(B, l + 2)) continue;
      a.step = 0;
      a.level += w < kSolve ? 2 : w < kSolve + kRing ? kRing : 1;
      if (a.level >= nlev) a.level = nlev, ++finished;
    }
    idle = 0;
  }
  CHECK(flight.empty());
}

int main() {
  int plans = 0;
  std::mt19937 rng(7);
  // random graphs of degree <= 4 on a strip (neighbours mostly close in the
  // elimination order, some far), all cluster sizes, down to one row
  for (int trial = 0; trial < 60; ++trial) {
    const int64_t sizes[] = {1, 2, 31, 32, 33, 63, 64, 65, 200, 1000, 5000, 20011};
    const int64_t n = sizes[trial % 12];
    const int width = 1 + (int)(rng() % 90);
    std::vector<int32_t> order(n), pos(n), nbr(4 * n, -1), deg(n, 0);
    for (int64_t i = 0; i < n; ++i) order[i] = (int32_t)i;
    if (trial % 3 == 0) std::shuffle(order.begin(), order.end(), rng);
    for (int64_t i = 0; i < n; ++i) pos[order[i]] = (int32_t)i;
    auto link = [&](int64_t i, int64_t k) {
      const int32_t a = order[i], b = order[k];
      if (a == b || deg[a] >= 4 || deg[b] >= 4) return;
      if (trial % 7 != 3)  // cells that share two edges otherwise
        for (int s = 0; s < 4; ++s)
          if (nbr[s * n + a] == b) return;
      int sa = (int)(rng() % 4), sb = (int)(rng() % 4);
      while (nbr[sa * n + a] >= 0) sa = (sa + 1) % 4;
      while (nbr[sb * n + b] >= 0) sb = (sb + 1) % 4;
      nbr[sa * n + a] = b;
      nbr[sb * n + b] = a;
      ++deg[a];
      ++deg[b];
    };
    for (int64_t i = 1; i < n; ++i) {
      if (trial % 5 != 4) link(i, std::max<int64_t>(0, i - width));
      if (rng() % 2) link(i, i - 1 - (int64_t)(rng() % std::min<int64_t>(i, width)));
      if (rng() % 20 == 0) link(i, (int64_t)(rng() % i));
    }
    for (int cluster : {0, 1, 2, 4, 8}) {
      const SweepPlan pl = make_sweep_plan(n, nbr, pos, order, cluster);
      if (pl.cluster == 0) {  // out of operand slots: only where long links are many
        CHECK(n >= 5000);
        continue;
      }
      ++plans;
      CHECK(pl.cluster <= kSweepMaxCluster);
      for (int dir = 0; dir < 2; ++dir) {
        walk(pl, dir, n, nbr, pos);
        if (n <= 5000 && cluster >= 0) simulate(pl, dir, n, nbr, pos, rng);
      }
    }
  }
  CHECK(plans >= 200);
  std::printf("ok %d\n", plans);
  return 0;
}
