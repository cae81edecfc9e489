// Host check of mge::soft::quot and mulquot against the host's arithmetic, bit for bit.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "soft_quotient_check.h"

using namespace mge::soft;

static bool same(double x, double y) { return (isnan(x) && isnan(y)) || bits(x) == bits(y); }

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  const double edge[] = {0.0, -0.0, 1.0, -1.0, 3.0, INFINITY, -INFINITY, NAN, 4.9406564584124654e-324,
                         2.2250738585072014e-308, 1.7976931348623157e308, 1.0000000000000002, 0.99999999999999989, 1e-300};
  long bad = 0, cases = 0;
  auto one = [&](double a, double b, double d) {
    const Recip R = recip(d);
    volatile double va = a, vb = b, vd = d, p = va * vb;
    cases++;
    if (same(quot(a, R, d), va / vd) && same(mulquot(a, b, R, d), p / vd)) return;
    if (bad++ < 10) printf("mismatch a=%a b=%a d=%a: %a/%a %a/%a\n", a, b, d, quot(a, R, d), va / vd, mulquot(a, b, R, d), p / vd);
  };
  for (double a : edge)
    for (double b : edge)
      for (double d : edge) one(a, b, d);
  for (int kind = 0; kind < 8; kind++)
    for (long i = 0; i < n; i++) {
      double a, b, d;
      triple(kind, (uint64_t)i, a, b, d);
      one(a, b, d);
    }
  printf("cases %ld mismatches %ld\n", cases, bad);
  return bad ? 1 : 0;
}
