// quick_quotient.h -- division by a divisor known in advance as one product and
// one fused multiply-add, with the host's check that it rounds as the division.
#pragma once
#include <cmath>
#include <cstdint>
#include <vector>

namespace mge {

// The low part yl of 1/y, yh = RN(1/y), for which fma(x, yh, RN(x*yl)) is the
// correctly rounded x/y for every finite x (products and quotient in the normal
// range): N. Brisebarre, J.-M. Muller, S. K. Raina, Accelerating correctly
// rounded floating-point division when the divisor is known in advance, IEEE
// Trans. Computers 53(8), 2004.  The value before the last rounding is within
// 2^-105 of x/y (significands in [1, 2)), so only an x whose quotient lies that
// near a midpoint M/2^s of two doubles can round wrongly.  With X, Y the
// integer significands, 2^s X - M Y is then a small integer r; for each r that
// fixes M, and so X, modulo a power of two, and the few X it leaves are tried
// against the division.  |r| <= 8 covers more than the bound asks for.  False
// when neither yl nor its neighbours pass.
inline bool quick_quotient(double y, double yh, double* low) {
  int e;
  const uint64_t Y = (uint64_t)std::ldexp(std::frexp(y, &e), 53);  // [2^52, 2^53)
  int g = 0;
  while (!((Y >> g) & 1)) g++;
  const uint64_t Yo = Y >> g;
  uint64_t inv = Yo;  // Yo^-1 modulo 2^64 by Newton's iteration
  for (int q = 0; q < 6; q++) inv *= 2 - Yo * inv;
  const uint64_t lo = 1ull << 52, hi = 1ull << 53;
  std::vector<double> xs;
  for (int s = 53; s <= 54; s++)
    for (int r = -8; r <= 8; r++) {
      if (r == 0 || g > 3 || r % (1 << g) != 0) continue;  // 2^g divides r
      // M Yo = -r / 2^g modulo 2^(s-g), M an odd integer of 54 bits
      const uint64_t mod = 1ull << (s - g), M0 = (uint64_t)(-(int64_t)(r / (1 << g))) * inv & (mod - 1);
      for (uint64_t M = M0 + ((hi - M0 + mod - 1) / mod) * mod; M < 2 * hi; M += mod) {
        if (!(M & 1)) continue;
        const unsigned __int128 n = (unsigned __int128)M * Y + (__int128)r;
        const uint64_t X = (uint64_t)(n >> s);
        if (((n >> s) << s) == n && X >= lo && X < hi) xs.push_back((double)X);
      }
    }
  const double yl0 = std::fma(-yh, y, 1.0) / y;  // the residual is exact
  for (int k = 0; k < 7; k++) {
    double yl = yl0;
    for (int q = 0; q < (k + 1) / 2; q++) yl = std::nextafter(yl, k & 1 ? -1.0 : 1.0);
    bool ok = true;
    for (double x : xs) ok = ok && std::fma(x, yh, x * yl) == x / y;
    if (ok) {
      *low = yl;
      return true;
    }
  }
  return false;
}

}  // namespace mge
