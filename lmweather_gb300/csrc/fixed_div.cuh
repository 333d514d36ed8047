// Correctly rounded division by a divisor fixed for a run (FP64), shared by the plane stencil and the FP64
// sphere synthesis.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <initializer_list>

namespace lmw {

constexpr unsigned long long kDivAbs = 0x7fffffffffffffffull, kDivMant = 0x000fffffffffffffull;

// x / y correctly rounded (round to nearest even), for a divisor y fixed for the run. GB300's FP64 pipe is narrow
// and an IEEE division costs several FP64 operations with a reciprocal seed; this costs three. The host stores the
// reciprocal as an unevaluated sum zh + zl (zh = RN(1/y), zl = RN(1/y - zh), formed exactly with an FMA), and
// q = RN(x zh + RN(x zl)) approximates x / y to about 2^-105 relative (the fixed-divisor scheme of N. Brisebarre,
// J.-M. Muller and S. K. Raina, "Accelerating correctly rounded floating-point division when the divisor is known
// in advance", IEEE Trans. Computers 53(8), 2004). q is ACCEPTED only on a proof that it is the rounded quotient:
// with gap the distance from |q| to the next double toward zero (the smaller of its two neighbour gaps) and
// T = |y| gap / 2 (a power-of-two scaling of y, formed exactly on the integer pipe), the FMA residual
// r = RN(x - q y) satisfies |r| < T only if |x - q y| < T (rounding is monotone and T is a double), that is
// |x / y - q| < gap / 2, which puts x / y strictly inside q's rounding interval. Zero dividends give the signed
// zero directly; everything else that is not accepted (ties, non-finite values, quotients or bounds outside the
// normal range) takes the IEEE division, so the result is RN(x / y) for every x.
__device__ __forceinline__ double div_fixed(double x, double y, double zh, double zl, int &fast) {
  const double q = __fma_rn(x, zh, __dmul_rn(x, zl));
  const double r = __fma_rn(-q, y, x);
  const unsigned long long bx = static_cast<unsigned long long>(__double_as_longlong(x));
  const unsigned long long by0 = static_cast<unsigned long long>(__double_as_longlong(y));
  const unsigned long long bq = static_cast<unsigned long long>(__double_as_longlong(q)) & kDivAbs;
  const unsigned long long by = by0 & kDivAbs;
  const unsigned long long br = static_cast<unsigned long long>(__double_as_longlong(r)) & kDivAbs;
  if ((bx & kDivAbs) == 0) {
    fast = 1;
    return __longlong_as_double(static_cast<long long>((bx ^ by0) & ~kDivAbs));
  }
  const int eq = static_cast<int>(bq >> 52);
  // biased exponent of T: |y| times 2^(exponent of gap - 1), gap = ulp(q), halved when q is a power of two
  const int et = static_cast<int>(by >> 52) + eq - 1023 - 53 - ((bq & kDivMant) == 0 ? 1 : 0);
  if (eq >= 1 && eq <= 2046 && et >= 1 && et <= 2046 &&
      br < ((static_cast<unsigned long long>(et) << 52) | (by & kDivMant))) {
    fast = 1;
    return q;
  }
  fast = 0;
  return x / y;
}

// the two-term reciprocal div_fixed needs: zh = RN(1/y), zl = RN(1/y - zh) (1 - y zh is exact for zh = RN(1/y), so
// the FMA forms it without error and the division rounds 1/y - zh once); false when y or zh is not a normal number
// (then divide plainly). A subnormal zl (|y| above about 2^969) only makes the fast path's answer rarer: the
// acceptance test does not depend on it.
inline bool fixed_div_reciprocal(double y, double &zh, double &zl) {
  zh = 1.0 / y;
  zl = std::fma(-y, zh, 1.0) / y;
  return std::fpclassify(y) == FP_NORMAL && std::fpclassify(zh) == FP_NORMAL && std::isfinite(zl);
}

// The same quotient in two FP64 operations, for divisors for which that is proven: q = RN(x zh + RN(x zl)) without
// div_fixed's residual. zh is 1/y rounded toward zero and zl >= 0 the rest, rounded and moved by `adj` units in its
// last place, so x zh + RN(x zl) is within (1 + |adj|) 2^-104 |x / y| of x / y, and q can differ from RN(x / y) only
// where x / y lies that close to the midpoint M of two neighbouring doubles. Scaled to integers X, Y in [2^52, 2^53)
// and an odd M this reads |2^k X - M Y| <= 8 (1 + |adj|) (k = 53 for X >= Y, else 54): for each of the few residues r the congruence 2^k X = r (mod Y) has one solution modulo the odd part of Y, so the
// host lists every fraction X that can go wrong and divides them all. A divisor is taken when at most one of them fails
// (for some adj); that one's 52 fraction bits are stored and take the IEEE division. Of 48,000 divisors of the form
// L / n and their squares all qualify, 93.6 % with no exception.
struct FixedDiv2 {
  double zh = 0, zl = 0;
  unsigned bad_hi = 0xffffffffu, bad_lo = 0;  // fraction bits of the exceptional dividend (bad_hi past 20 bits: none)
};

// x / y by f; ok = 0 when the caller has to divide: exponents outside 2^-800 .. 2^800 (products that could leave the
// normal range, infinities, NaN) and the exceptional fraction. Zeros pass (zh > 0 and zl >= 0 keep the sign).
__device__ __forceinline__ double div_fixed2(double x, const FixedDiv2 &f, int &ok) {
  const double q = __fma_rn(x, f.zh, __dmul_rn(x, f.zl));
  const unsigned hi = static_cast<unsigned>(__double2hiint(x)), lo = static_cast<unsigned>(__double2loint(x));
  const unsigned a = hi & 0x7fffffffu;
  const bool in = a - (223u << 20) < (1600u << 20) || (a | lo) == 0u;
  ok = in && !((hi & 0xfffffu) == f.bad_hi && lo == f.bad_lo) ? 1 : 0;
  return q;
}

// the parameters of div_fixed2 for y, or false when no zl makes all but one dividend provably right (or y is not a
// positive number between 2^-100 and 2^100)
inline bool fixed_div2_setup(double y, FixedDiv2 &out) {
  if (!(y >= 0x1p-100 && y <= 0x1p100)) return false;
  int ex = 0;
  const uint64_t Y = static_cast<uint64_t>(std::ldexp(std::frexp(y, &ex), 53));
  const double ys = static_cast<double>(Y);
  int t = 0;
  uint64_t Yo = Y;
  while (!(Yo & 1)) {
    Yo >>= 1;
    t++;
  }
  uint64_t yinv = Yo;  // Yo^-1 mod 2^64 (Newton: each step doubles the correct bits, three to start with)
  for (int i = 0; i < 5; i++) yinv *= 2 - Yo * yinv;
  double zh = 1.0 / ys;
  if (std::fma(-ys, zh, 1.0) < 0) zh = std::nextafter(zh, 0.0);
  const double rest = std::fma(-ys, zh, 1.0) / ys;  // exact remainder, rounded quotient
  for (int adj : {0, 1, -1, 2, -2, 3, -3, 4, -4}) {
    double zl = rest;
    for (int k = 0; k < std::abs(adj); k++) zl = std::nextafter(zl, adj > 0 ? 1.0 : 0.0);
    if (rest == 0 && adj != 0) break;
    int bad = 0;
    uint64_t bad_x = 0;
    auto check = [&](uint64_t x) {  // every X congruent to x
      if (x < (1ull << 52)) x += ((1ull << 52) - x + Yo - 1) / Yo * Yo;
      for (; x < (1ull << 53); x += Yo) {
        const double xs = static_cast<double>(x);
        if (std::fma(xs, zh, xs * zl) != xs / ys && x != bad_x) {
          bad++;
          bad_x = x;
        }
      }
    };
    for (int k = 53; k <= 54 && t <= 6; k++) {
      // 2^-(k - t) mod Yo = (1 + Yo m) / 2^(k - t) with m = -Yo^-1 mod 2^(k - t); r is a multiple of 2^t
      const uint64_t m = (0 - yinv) & ((1ull << (k - t)) - 1);
      const uint64_t inv = static_cast<uint64_t>((static_cast<unsigned __int128>(Yo) * m + 1) >> (k - t)) % Yo;
      uint64_t x = 0;
      for (int r = 1; r <= (8 * (1 + std::abs(adj))) >> t; r++) {
        x = x + inv >= Yo ? x + inv - Yo : x + inv;
        check(x);
        check(Yo - x);
      }
    }
    if (bad > 1) continue;
    out.zh = std::ldexp(zh, 53 - ex);
    out.zl = std::ldexp(zl, 53 - ex);
    out.bad_hi = bad ? static_cast<unsigned>(bad_x >> 32) & 0xfffffu : 0xffffffffu;
    out.bad_lo = bad ? static_cast<unsigned>(bad_x) : 0u;
    return true;
  }
  return false;
}

}  // namespace lmw
