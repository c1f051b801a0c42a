// CPU check of o2f::recip_seeded, o2f::quot and o2f::sqrt_seeded (csrc/qdiv.h): with any seed
// within 2^-18 the reciprocal is RN(1/b), the quotient RN(a/b) and the root
// RN(sqrt(a)), bit for bit, unless `ok` is cleared -- and it is cleared only outside the
// stated range.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>

#include "qdiv.h"

static uint64_t g = 88172645463325252ull;
static uint64_t rnd() {
  g ^= g << 13;
  g ^= g >> 7;
  return g ^= g << 17;
}
static double make(int emin, int emax) {
  uint64_t u = (rnd() & ((1ull << 52) - 1)) | ((uint64_t)(1023 + emin + (int)(rnd() % (emax - emin + 1))) << 52) |
               ((rnd() & 1) << 63);
  if (rnd() % 4 == 0) u |= ((1ull << 52) - 1) & ~((1ull << (rnd() % 40)) - 1);  // significands near all ones
  if (rnd() % 8 == 0) u &= ~((1ull << (rnd() % 52)) - 1);                       // short significands
  double x;
  std::memcpy(&x, &u, 8);
  return x;
}
static bool same(double x, double y) { return std::memcmp(&x, &y, 8) == 0; }

int main() {
  long bad = 0, refused = 0;
  const long n = 6000000;
  for (long i = 0; i < n; ++i) {
    const double b = make(-60, 60);
    double a = make(-60, 60);
    if (i % 16 == 0) a = (rnd() & 1) ? 0.0 : -0.0;
    if (i % 16 == 1) a = b * make(-2, 2);  // quotients of few bits
    const double seed = (1.0 / b) * (1.0 + (double)((int64_t)(rnd() % 2001) - 1000) / 1000.0 * 0x1p-18);
    bool ok = true;
    const double y = o2f::recip_seeded(b, seed, ok);
    if (!ok) {
      uint64_t u;
      std::memcpy(&u, &b, 8);
      if ((u & ((1ull << 52) - 1)) != (1ull << 52) - 1) ++bad;  // refused without a reason
      ++refused;
      continue;
    }
    if (!same(y, 1.0 / b)) ++bad;
    const double q = o2f::quot(a, b, y, ok);
    if (!ok || !same(q, a / b)) ++bad;
    const double c = std::fabs(i % 3 ? a : q * q * (1.0 + (double)(i % 5 - 2) * 0x1p-52));  // near squares too
    const double rs = 1.0 / std::sqrt(c) * (1.0 + (double)((int64_t)(rnd() % 2001) - 1000) / 1000.0 * 0x1p-18);
    bool k1 = true;
    const double root = o2f::sqrt_seeded(c, rs, k1);
    if (k1 ? !same(root, std::sqrt(c)) : c != 0.0) ++bad;
    // out of range: refused, not wrong
    const double big = make(-1000, 1000), small = make(-1000, 1000);
    bool k2 = true;
    const double y2 = o2f::recip_seeded(small, 1.0 / small, k2);
    const double q2 = k2 ? o2f::quot(big, small, y2, k2) : 0.0;
    if (k2 && !same(q2, big / small)) ++bad;
  }
  const double special[] = {INFINITY, -INFINITY, NAN, 0.0, -0.0, 5e-324, 1e308, 0x1p-1022};
  for (double b : special)
    for (double a : {1.0, 0.0, -0.0, 1e300, 5e-324, (double)INFINITY, (double)NAN}) {
      bool ok = true;
      const double y = o2f::recip_seeded(b, 1.0 / b, ok);
      if (ok) ++bad;  // none of these divisors is in range
      bool k = true;
      const double q = o2f::quot(a, 3.0, 1.0 / 3.0, k);
      if (k && !same(q, a / 3.0)) ++bad;
      (void)y;
    }
  std::printf("%ld operands, %ld refused, %ld wrong\n", n, refused, bad);
  return bad ? 1 : 0;
}
