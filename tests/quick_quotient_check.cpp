// Checks quick_quotient.h: for the pivots of the line sweeps at many smoothing
// coefficients and for random divisors, every quotient formed with the low part
// it accepts equals the division, on random dividends and on those whose
// quotients lie next to a midpoint of two doubles, where a wrong rounding would
// have to be.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "quick_quotient.h"

static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { return s ^= s << 13, s ^= s >> 7, s ^= s << 17; }
static double sig(uint64_t r) {  // a double in [1, 2)
  const uint64_t u = (r >> 12) | 0x3ff0000000000000ull;
  double x;
  memcpy(&x, &u, 8);
  return x;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 20000;
  long bad = 0, refused = 0, divisors = 0;
  auto check = [&](double y) {
    const double yh = 1.0 / y;
    double yl;
    divisors++;
    if (!mge::quick_quotient(y, yh, &yl)) {
      refused++;
      return;
    }
    auto one = [&](double x) { bad += std::fma(x, yh, x * yl) != x / y; };
    for (long q = 0; q < n; q++) {
      one(std::ldexp(sig(rnd()), (int)(rnd() % 600) - 300) * (rnd() & 1 ? 1.0 : -1.0));
      // a dividend next to y times a midpoint: the quotient almost a tie
      const double m = sig(rnd()), h = std::ldexp(1.0, -53);
      double x = (double)((long double)y * ((long double)m + (long double)h));
      one(x);
      one(std::nextafter(x, 0.0));
      one(std::nextafter(x, 1e300));
    }
  };
  for (int k = 0; k < 40; k++) {
    const double smoo = k == 0 ? 0.6 : 0.05 * k, aa = 1.0 + 2.0 * smoo, bb = -smoo;
    double e1 = aa, e2 = bb / aa, last = 0.0;
    for (int q = 0; q < 64 && e1 != last; q++) {
      check(e1);
      last = e1;
      e1 = aa - bb * e2;
      e2 = bb / e1;
    }
  }
  for (int q = 0; q < 300; q++) check(sig(rnd()) * (1 << rnd() % 4));
  for (int g = 1; g < 8; g++) check(sig(rnd() & (~0ull << (12 + g))));  // trailing zeros
  printf("divisors %ld refused %ld bad %ld\n", divisors, refused, bad);
  return bad != 0 || refused * 50 > divisors;
}
