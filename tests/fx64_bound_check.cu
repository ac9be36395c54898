// Host-side check of fx64.cuh's bound of a held value, run by tests/test_fx64_bound_host.py:
// cterm is above |re| + |im| in its unit for every shift, and by less than 2 units;
// 256 of the largest fit 32 bits.
#include <cstdio>
#include <random>

#include "fx64.cuh"

using namespace nhqg::fx;

int main() {
  std::mt19937_64 g(11);
  long bad = 0;
  const long long ones = (1LL << 40) - 1;
  for (int i = 0; i < 400000; ++i) {
    const int bits = 62 - (int)(g() % 50);
    auto part = [&] {
      long long v = (long long)(g() >> 2) & ((1LL << bits) - 1);
      if (i & 1) v |= ones;  // the largest remainder below the unit
      return (g() & 1) ? -v : v;
    };
    const cfx z{part(), part()};
    const int sh = (int)(g() % 32);
    const long double unit = (long double)(1LL << 40) * (long double)(1LL << sh);
    const long double v = (long double)(z.x < 0 ? -z.x : z.x) + (long double)(z.y < 0 ? -z.y : z.y);
    const long double t = (long double)cterm(z, sh) * unit;
    if (!(t > v) || !(t - v <= 2.0L * unit)) ++bad;
  }
  const long long top = (1LL << 62) - 1;
  if (256ull * cterm(cfx{top, -top}, 0) >= (1ull << 32)) ++bad;
  if (cterm(cfx{0, 0}, 0) != 2u || cterm(cfx{0, 0}, 5) != 1u) ++bad;
  std::printf("bad %ld\n", bad);
  return bad == 0 ? 0 : 1;
}
