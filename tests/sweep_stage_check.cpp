// Host check of the block ILU sweeps' data path: the factor blocks as
// k_ilu_pack writes them, the copies of a level into shared memory as the
// staging warps start them, and what load_row reads there (and a fourth
// dependency's blocks from global memory), with a tag for each element.  Every
// read finds its own element, every copy and read stays inside its buffer.
// The layout's constants come from ilu.cuh (the build's -D options).
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

constexpr int kStageRing = STAGE_RING, kStageChunkDoubles = STAGE_CHUNK, kStageBwdD = STAGE_BWD_D,
              kStageDoubles = STAGE_DOUBLES, kStageOwn = STAGE_OWN;

static double tag_of_block(int row, int slot, int el) { return 80.0 * row + 16 * (1 + slot) + el; }
static double tag_of_inverse(int row, int el) { return -(16.0 * row + el) - 1.0; }

static void check(const SweepPlan& pl, int dir, int64_t n, const std::vector<int32_t>& nbr,
                  const std::vector<int32_t>& pos) {
  const int C = pl.cluster;
  const auto &rec = pl.rec[dir], &info = pl.info[dir];
  const int64_t chunks = pl.chunks[dir];
  // k_ilu_pack, a thread per pair of doubles
  std::vector<double> pack(chunks * 2048, 0.5), packD(chunks * 512, 0.5), own(chunks * 128);
  for (int64_t i = 0; i < chunks * 128; ++i) own[i] = 1e9 + (double)i;
  for (int inverse = 0; inverse < 2; ++inverse) {
    const int per = inverse ? 256 : 1024;
    for (int64_t t = 0; t < chunks * per; ++t) {
      const int64_t chunk = t / per;
      const int d = (int)(t % per) >> 8, in = (int)(t & 255), half = in >> 7, q = (in >> 2) & 31, c = in & 3;
      const int32_t* r = rec.data() + (chunk * 32 + q) * kSweepRec;
      if (r[0] < 0 || (!inverse && d >= r[1])) continue;
      const int slot = (int)(((uint32_t)r[9] >> (8 * (d & 3))) & 0xff);
      double* dst = inverse ? packD.data() + chunk * 512 : pack.data() + chunk * 2048 + d * 512;
      for (int e = 0; e < 2; ++e) {
        double& x = dst[sweep_pack_place(q, 4 * c + 2 * half) + e];
        CHECK(x == 0.5);  // written once
        const int el = 4 * c + 2 * half + e;
        x = inverse ? tag_of_inverse(r[0], el) : tag_of_block(r[0], slot, el);
      }
    }
  }
  std::vector<double> blk(kStageRing * kStageDoubles, 0.25), s_own(kStageRing * kStageOwn, 0.25);
  int64_t rows = 0;
  auto copy = [](std::vector<double>& to, int64_t at, int64_t end, const std::vector<double>& from, int64_t src, int bytes) {
    CHECK(at % 2 == 0 && src % 2 == 0 && bytes % 16 == 0);
    CHECK(at >= 0 && at + bytes / 8 <= end && src >= 0 && src + bytes / 8 <= (int64_t)from.size());
    std::copy(from.begin() + src, from.begin() + src + bytes / 8, to.begin() + at);
  };
  for (int l = 0; l < pl.nlev[dir]; ++l) {
    const int slot = l % kStageRing;
    for (int b = 0; b < C; ++b) {
      const int32_t* in = info.data() + ((size_t)l * C + b) * 4;
      for (int j = 0; j < in[1]; ++j) {
        const int64_t k = in[0] + (int64_t)j * C, base = (int64_t)slot * kStageDoubles;
        copy(blk, base + j * kStageChunkDoubles, base + (j + 1) * kStageChunkDoubles, pack, k * 2048,
             (in[2] >> j & 1 ? 3 : 2) * 4096);
        if (dir == 1) copy(blk, base + kStageBwdD + j * 512, base + kStageDoubles, packD, k * 512, 4096);
        copy(s_own, (int64_t)slot * kStageOwn + j * 128, (int64_t)(slot + 1) * kStageOwn, own, k * 128, 1024);
      }
      // load_row: four lanes a row
      for (int j = 0; j < in[1]; ++j)
        for (int w = 0; w < 4; ++w)
          for (int lane = 0; lane < 32; ++lane) {
            const int q = w * 8 + (lane >> 2), c = lane & 3;
            const int64_t k = in[0] + (int64_t)j * C, p = k * 32 + q;
            const int32_t* r = rec.data() + p * kSweepRec;
            if (r[0] < 0) continue;
            rows += c == 0;
            const double* s = blk.data() + slot * kStageDoubles + (q * 4 + c) * 2;
            CHECK(s_own[slot * kStageOwn + j * 128 + q * 4 + c] == own[4 * p + c]);
            if (dir == 1)
              for (int e = 0; e < 4; ++e)
                CHECK(s[kStageBwdD + j * 512 + (e >> 1) * 256 + (e & 1)] == tag_of_inverse(r[0], 4 * c + e));
            int d = 0;
            for (int sl = 0; sl < 4; ++sl) {
              const int32_t o = nbr[sl * n + r[0]];
              if (o < 0 || !(dir == 0 ? pos[o] < pos[r[0]] : pos[o] > pos[r[0]])) continue;
              for (int e = 0; e < 4; ++e) {
                const int at = (e >> 1) * 256 + (e & 1);
                const double v = d < 3 ? s[j * kStageChunkDoubles + d * 512 + at]
                                       : pack[k * 2048 + 1536 + (q * 4 + c) * 2 + at];
                CHECK(v == tag_of_block(r[0], sl, 4 * c + e));
              }
              ++d;
            }
            CHECK(d == r[1]);
          }
    }
  }
  CHECK(rows == n);
}

int main() {
  std::mt19937 rng(5);
  int fourth = 0;
  for (int trial = 0; trial < 24; ++trial) {
    const int64_t sizes[] = {1, 33, 64, 65, 500, 4000};
    const int64_t n = sizes[trial % 6];
    const int width = 2 + (int)(rng() % 70);
    std::vector<int32_t> order(n), pos(n), nbr(4 * n, -1);
    for (int64_t i = 0; i < n; ++i) order[i] = (int32_t)i;
    std::shuffle(order.begin(), order.end(), rng);
    for (int64_t i = 0; i < n; ++i) pos[order[i]] = (int32_t)i;
    auto link = [&](int64_t i, int64_t k) {
      if (k < 0 || i == k) return;
      const int32_t a = order[i], b = order[k];
      int sa = (int)(rng() % 4), sb = (int)(rng() % 4), m = 0;
      while (m < 4 && nbr[((sa + m) % 4) * n + a] >= 0) ++m;
      sa = (sa + m) % 4;
      if (m == 4) return;
      for (m = 0; m < 4 && nbr[((sb + m) % 4) * n + b] >= 0;) ++m;
      sb = (sb + m) % 4;
      if (m == 4) return;
      nbr[sa * n + a] = b;
      nbr[sb * n + b] = a;
    };
    for (int64_t i = 1; i < n; ++i) {
      link(i, i - width);
      for (int t = 0; t < 3; ++t)
        if (rng() % 3 == 0) link(i, i - 1 - (int64_t)(rng() % width));
    }
    for (int cluster : {1, 2, 4, 8}) {
      const SweepPlan pl = make_sweep_plan(n, nbr, pos, order, cluster);
      if (pl.cluster == 0) continue;
      for (int dir = 0; dir < 2; ++dir) {
        check(pl, dir, n, nbr, pos);
        for (size_t p = 0; p < pl.rec[dir].size(); p += kSweepRec) fourth += pl.rec[dir][p] >= 0 && pl.rec[dir][p + 1] == 4;
      }
    }
  }
  CHECK(fourth > 0);
  std::printf("ok %d\n", fourth);
  return 0;
}
