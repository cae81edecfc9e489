// Operand triples for mge::soft::quot and mulquot, shared by the host and the
// device check: any bit patterns, moderate exponents, products and quotients
// near underflow and overflow, the magnitudes of a flow solver, divisors with a
// significand at or next to 1 or 2, short significands (exact products, ties),
// and dividends next to an exact quotient or to a midpoint of two.
#pragma once
#include "soft_fp64.cuh"

MGE_SF_HD uint64_t mix64(uint64_t x) {  // splitmix64 finaliser
  x ^= x >> 30;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 27;
  x *= 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
MGE_SF_HD double draw_exp(uint64_t r, uint64_t e) {
  return mge::soft::from_bits((r & (mge::soft::kFrac | mge::soft::kSign)) | (e << 52));
}
MGE_SF_HD void triple(int kind, uint64_t i, double& a, double& b, double& d) {
  using namespace mge::soft;
  const uint64_t r1 = mix64(4 * i + 1), r2 = mix64(4 * i + 2), r3 = mix64(4 * i + 3), r4 = mix64(i ^ 0x5bd1e995ull);
  a = draw_exp(r1, 1013 + r4 % 21), b = draw_exp(r2, 1003 + (r4 >> 7) % 31), d = draw_exp(r3, 1018 + (r4 >> 20) % 10);
  if (kind == 0) a = from_bits(r1), b = from_bits(r2), d = from_bits(r3);
  if (kind == 1) a = draw_exp(r1, 1 + r4 % 2046), b = draw_exp(r2, 1 + (r4 >> 12) % 2046), d = draw_exp(r3, 1 + (r4 >> 24) % 2046);
  if (kind == 2) a = draw_exp(r1, 1 + r4 % 600), b = draw_exp(r2, 430 + (r4 >> 12) % 600);
  if (kind == 3) {
    const uint64_t low = (r3 >> 1) % 4096;
    d = from_bits(((1000 + (r4 >> 9) % 40) << 52) | ((r3 & 1) ? low : kFrac - low));
  }
  if (kind == 4) a = from_bits(bits(a) & ~0xFFFFFFFFFFull), b = from_bits(bits(b) & ~0xFFFFFFFull);
  if (kind == 5) {  // (a b) next to d times a short significand: quotients a few ulps from exact
    b = 1.0;
    a = from_bits(bits(mul(d, from_bits(bits(draw_exp(r1, 1015 + r4 % 16)) & ~0xFFFFFFFFFull))) + (r4 >> 40) % 5 - 2);
  }
  if (kind == 6) {  // ... next to d times a midpoint: quotients a few ulps of the dividend from halfway
    b = 1.0;
    const uint64_t q = (r1 & kFrac) | kOne, dm = bits(d) & kFrac;  // d (q + 1/2) in integers, high part
    const uint64_t D = dm | kOne, t = mulhi64(D << 11, (2 * q + 1) << 10);
    a = from_bits(((t >> 52 ? t >> 1 : t) & kFrac) | (1023ull << 52));
    a = from_bits(bits(a) + (r4 >> 40) % 5 - 2);
  }
}
