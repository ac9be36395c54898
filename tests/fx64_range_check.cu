// Host-side check of fx64.cuh's products at the end of their range, run by
// tests/test_fx64_range_host.py: values of modulus up to 2^62, twice what sequences
// from FP64 hold.  Bounds in units: a component of a complex product joins two partial
// products (at most 2 each dropped, 4), one rounding (1/2) and twiddle factors rounded by
// 1/2 (c) against |x + y| <= 2^1.5 and by 1 (s - c, s + c) against |x|, |y| <= 2, in units of
// 2^61: 1.5 + 2.  In all 8.  A real product: 2 + 1/2 + 1/2 2^1.5 = 4; the rotations by pi/4
// are real products of a sum.  A shifted product (rs >= 62): its dropped low x low, at
// most 2^62 / 2^rs, a rounding and a floor, within the 3.5 of fx64_check.cu.
#include <cmath>
#include <cstdio>
#include <random>

#include "fx64.cuh"

using namespace nhqg::fx;

int main() {
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  const long double one = std::ldexp(1.0L, kBits), top = std::ldexp(1.0L, 62) * (1.0L - 1e-6L);
  const long double pi = 3.14159265358979323846264338327950288L;
  double w_cmul = 0, w_rot = 0, w_real = 0, w_mul = 0;
  for (int i = 0; i < 400000; ++i) {
    // on the circle of modulus 2^62, at the diagonals and axes every other time
    const long double ph = i & 1 ? pi * u(g) : pi / 4 * (int)(g() % 8);
    const cfx a{(long long)(top * std::cos(ph)), (long long)(top * std::sin(ph))};
    const long double t = pi * u(g);
    const long long c = std::llround(std::cos(t) * one), s = std::llround(std::sin(t) * one);
    const Tw w = make_tw(c, s);
    const long double cl = std::cos(t), sl = std::sin(t);
    const cfx p = cmul<false>(a, w), q = cmul<true>(a, w);
    const long double e[4] = {p.x - (a.x * cl - a.y * sl), p.y - (a.x * sl + a.y * cl),
                              q.x - (a.x * cl + a.y * sl), q.y - (a.y * cl - a.x * sl)};
    for (long double v : e) w_cmul = std::max(w_cmul, (double)std::fabs(v));
    auto rerr = [&](cfx z, long double th) {
      const long double cc = std::cos(th), ss = std::sin(th);
      w_rot = std::max(w_rot, (double)std::fabs(z.x - (a.x * cc - a.y * ss)));
      w_rot = std::max(w_rot, (double)std::fabs(z.y - (a.x * ss + a.y * cc)));
    };
    rerr(rot<8, 1, 1>(a), pi / 4);
    rerr(rot<8, 3, -1>(a), -3 * pi / 4);
    rerr(rot<12, 5, 1>(a), 5 * pi / 6);
    rerr(rot<16, 3, -1>(a), -3 * pi / 8);
    const long long h = sin48(16);
    w_real = std::max(w_real, (double)std::fabs(rmul(a.x, h) - a.x * std::sqrt(3.0L) / 2));
    const int rs = 62 + (int)(g() % 65);
    const __int128 f = (__int128)a.x * a.y;
    w_mul = std::max(w_mul, (double)std::fabs(mul_shift(a.x, a.y, rs) - (long double)f / std::ldexp(1.0L, rs)));
  }
  std::printf("cmul %.3f rot %.3f real %.3f mul %.3f\n", w_cmul, w_rot, w_real, w_mul);
  return w_cmul <= 8.0 && w_rot <= 8.0 && w_real <= 4.0 && w_mul <= 3.5 ? 0 : 1;
}
