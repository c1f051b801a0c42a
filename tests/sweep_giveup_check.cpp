// Host check of the block ILU sweeps when waits run out (k_ilu_sweep_cluster):
// the kernel's warps in random order, any of whose waits may give up, with
// some values held back.  Checked: a staged slot is never filled while a warp
// that has not given up reads it; no barrier is set, and none arrived on,
// beyond the phase that runs; all warps reach the end; nothing is on its way
// into a block that has no warp that gave up (such a block ends at once; one
// with such a warp waits).
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

struct Bar {
  int count, pending, done = 0;
  int64_t tx = 0;
  explicit Bar(int c) : count(c), pending(c) {}
  void settle() {
    if (pending == 0 && tx == 0) ++done, pending = count;
  }
  void arrive(int64_t expect) {
    CHECK(pending > 0);  // a phase takes no more arrivals than it waits for
    tx += expect;
    --pending;
    settle();
  }
  void complete(int64_t b) {
    tx -= b;
    settle();
  }
  bool passes(int phase) const { return (done & 1) != (phase & 1); }
};

static int simulate(const SweepPlan& pl, int dir, std::mt19937& rng, int held, int chance) {
  constexpr int kRing = 4, kWarps = 4 * kSweepChunks;
  constexpr int kSolve = 2 * kWarps, kAll = kSolve + kRing + 1;
  const int C = pl.cluster, nlev = pl.nlev[dir];
  const auto &info = pl.info[dir], &rec = pl.rec[dir];
  auto in = [&](int l, int b, int f) { return info[((size_t)l * C + b) * 4 + f]; };
  struct Block {
    std::vector<Bar> op, full, empty;
    std::vector<int> staged, readers;  // level in a slot; warps that read it now
    bool quit = false;
    Block() : op(kSweepBars, Bar(1)), full(kRing, Bar(1)), empty(kRing, Bar(kWarps)), staged(kRing, -1), readers(kRing, 0) {}
  };
  std::vector<Block> blk(C);
  struct Flight {
    int rank, bar;
  };
  std::vector<Flight> flight;
  struct Actor {
    int level = -1, step = 0, arrivals = 0;
    bool bad = false, reading = false, ended = false;
  };
  std::vector<Actor> act(C * kAll);
  auto all_arrived = [&](int k) {
    for (auto& a : act)
      if (a.arrivals < k) return false;
    return true;
  };
  // a wait: over, still on, or run out (then the warp is bad and goes on)
  auto wait = [&](Actor& a, Block& B, const Bar& bar, int phase) {
    if (a.bad || bar.passes(phase)) return true;
    if (B.quit || (int)(rng() % 1000) < chance) {
      a.bad = true;
      B.quit = true;
      return true;
    }
    return false;
  };
  auto stage = [&](Block& B, int l) {
    if (l >= nlev) return;
    CHECK(B.readers[l % kRing] == 0);
    B.staged[l % kRing] = l;
    B.full[l % kRing].arrive(0);
  };
  auto arm = [&](int b, int l) {
    if (l < nlev) blk[b].op[l % kSweepBars].arrive(in(l, b, 3));
  };
  // one step of taking a staged level's rows; true when it is done
  auto load = [&](Actor& a, Block& B, int l) {
    const int slot = l % kRing;
    if (!a.reading) {
      if (!wait(a, B, B.full[slot], l / kRing)) return false;
      if (!a.bad) {
        CHECK(B.staged[slot] == l);
        ++B.readers[slot];
        a.reading = true;
        return false;
      }
#ifdef BAD_WARPS_ARRIVE
      if (B.empty[slot].pending > 0) B.empty[slot].arrive(0);
#endif
      return true;
    }
    CHECK(B.staged[slot] == l);
    --B.readers[slot];
    a.reading = false;
    B.empty[slot].arrive(0);
    return true;
  };
  int64_t idle = 0;
  int finished = 0;
  while (finished < C * kAll) {
    CHECK(++idle < 4000000);
    if (!flight.empty() && rng() % 3 == 0) {
      const size_t i = rng() % flight.size();
      const Flight f = flight[i];
      flight[i] = flight.back();
      flight.pop_back();
      blk[f.rank].op[f.bar].complete(32);
      idle = 0;
    }
    const int who = (int)(rng() % act.size()), b = who / kAll, w = who % kAll;
    Actor& a = act[who];
    Block& B = blk[b];
    if (a.ended) continue;
    if (a.level >= nlev) {  // the last cluster barriers
      if (a.step < 2) ++a.arrivals, a.step = 2;
      else if (all_arrived((nlev + kSweepSkew / 2 - 1) / (kSweepSkew / 2) + 1)) a.ended = true, ++finished;
      idle = 0;
      continue;
    }
    if (a.level < 0) {
      if (w >= kSolve && w < kSolve + kRing) stage(B, w - kSolve);
      if (w == kSolve + kRing)
        for (int l = 0; l < kSweepNear; ++l) arm(b, l);
      if (w < kSolve && w / kWarps < nlev && !load(a, B, w / kWarps)) continue;
      a.level = 0;
      idle = 0;
      continue;
    }
    const int l = a.level + (w < kSolve ? w / kWarps : w < kSolve + kRing ? w - kSolve : 0);
    if (a.step == 0) {
      if (a.level % (kSweepSkew / 2) == 0) {
        if (a.level > 0 && !all_arrived(a.level / (kSweepSkew / 2))) continue;
        ++a.arrivals;
#ifndef ARM_UNSEEN
        if (w == kSolve + kRing && B.quit) a.bad = true;
#endif
      }
      a.step = 1;
    } else if (l >= nlev) {
      a.level = nlev;
      a.step = 0;
    } else if (a.step == 1) {
      if (w < kSolve) {
        if (!wait(a, B, B.op[l % kSweepBars], l / kSweepBars)) continue;
        const int j = w / 4 % kSweepChunks;
        if (!a.bad && j < in(l, b, 1)) {
          const int64_t k = in(l, b, 0) + (int64_t)j * C;
          for (int q = w % 4 * 8; q < w % 4 * 8 + 8; ++q) {
            const int32_t* r = rec.data() + (size_t)(k * 32 + q) * kSweepRec;
            if (r[0] < 0 || r[0] == held) continue;
            for (int t = 4; t < 8 && r[t] >= 0; ++t) flight.push_back({r[t] >> 16, r[t] >> 12 & 15});
          }
        }
      } else if (w < kSolve + kRing) {
        if (!wait(a, B, B.empty[l % kRing], l / kRing)) continue;
        if (!a.bad) stage(B, l + kRing);
      } else {
        if (!a.bad) arm(b, l + kSweepNear);
      }
      a.step = 2;
    } else {
      if (w < kSolve && l + 2 < nlev && !load(a, B, l + 2)) continue;
      a.step = 0;
      a.level += w < kSolve ? 2 : w < kSolve + kRing ? kRing : 1;
      if (a.level >= nlev) a.level = nlev;
    }
    idle = 0;
  }
  std::vector<char> bad(C, 0);
  int gave_up = 0;
  for (int i = 0; i < C * kAll; ++i) {
    bad[i / kAll] |= act[i].bad;
    gave_up += act[i].bad;
  }
  for (const Flight& f : flight) CHECK(bad[f.rank]);
  return gave_up;
}

int main() {
  std::mt19937 rng(11);
  int gave_up = 0, clean = 0, runs = 0;
  for (int trial = 0; trial < 24; ++trial) {
    const int64_t sizes[] = {1, 40, 200, 700, 1500, 3000};
    const int64_t n = sizes[trial % 6];
    const int width = 2 + (int)(rng() % 60);
    std::vector<int32_t> order(n), pos(n), nbr(4 * n, -1);
    for (int64_t i = 0; i < n; ++i) order[i] = pos[i] = (int32_t)i;
    auto link = [&](int64_t a, int64_t b) {
      if (a == b || b < 0) return;
      int sa = 0, sb = 0;
      while (sa < 4 && nbr[sa * n + a] >= 0) ++sa;
      while (sb < 4 && nbr[sb * n + b] >= 0) ++sb;
      if (sa == 4 || sb == 4) return;
      nbr[sa * n + a] = (int32_t)b;
      nbr[sb * n + b] = (int32_t)a;
    };
    for (int64_t i = 1; i < n; ++i) {
      link(i, i - width);
      if (rng() % 2) link(i, i - 1);
    }
    for (int cluster : {1, 2, 4, 8}) {
      const SweepPlan pl = make_sweep_plan(n, nbr, pos, order, cluster);
      if (pl.cluster == 0) continue;
      for (int dir = 0; dir < 2; ++dir) {
        const int kind = (int)(rng() % 3);  // values held back, waits that run out by themselves, neither
        const int got = simulate(pl, dir, rng, kind == 0 ? (int)(rng() % n) : -1, kind == 2 ? 0 : 1 + (int)(rng() % 4));
        ++runs;
        gave_up += got > 0;
        clean += got == 0;
      }
    }
  }
  CHECK(gave_up >= 40 && clean >= 20);
  std::printf("ok %d %d\n", gave_up, clean);
  return 0;
}
