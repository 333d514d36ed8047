// The butterfly of the FP64 grid stage's FFTs (sphere.cu) and its factors.
//
// Radix 2, decimation in time, one component c (0 real, 1 imaginary) of x = u + w v and y = u - w v a call. With the larger of
// the twiddle's cosine and sine taken out, w v = s (p + r q) for two of the components of v, the factor s and the ratio r of at most
// one (E. Linzer and E. Feig, "Implementation of efficient FFT algorithms on fused multiply-add architectures", IEEE Trans.
// Signal Processing 41(1), 1993): three FMAs instead of four operations, and u, mostly the larger, meets one rounding in x and
// one in y, as in separate sums. (Two FMAs around u and y = 2 u - x cost as little, but round at the size of u twice and give
// y the error of x: small wavenumbers beside a large mean had 1.25 to 1.45 times the error.) The first two stages have
// w = 1 and +-i and take two operations.
#pragma once
#include <cmath>

namespace lmw {

// factors of the stages 2 and up of a transform of n = 2^logn points: stage st's at t[2 (2^st + lo)], lo < 2^st: s, then r.
// Stage st has w = exp(-i pi lo / 2^st); angles are reduced to an eighth of a turn
inline void fft64_factors(int logn, double *t) {
  const double pi = 3.14159265358979323846;
  for (int k = 0; k < 8 && k < 2 << logn; k++) t[k] = 0;
  for (int st = 2; st < logn; st++) {
    const int h = 1 << st;
    for (int lo = 0; lo < h; lo++) {
      const bool by_sine = 4 * lo > h && 4 * lo < 3 * h;
      // from the nearest of 0, a quarter and half a turn (in the direction that keeps it in -1/8 .. 1/8)
      const int k = by_sine ? h / 2 - lo : 4 * lo <= h ? lo : h - lo;
      const double a = pi * k / h, tan = 4 * k == h ? 1.0 : 4 * k == -h ? -1.0 : std::tan(a);
      double *w = t + 2 * (h + lo);
      w[0] = by_sine || 4 * lo > h ? -std::cos(a) : std::cos(a);  // the sine of w is -sin, and -cos(a) past a quarter
      w[1] = by_sine || 4 * lo <= h ? -tan : tan;
    }
  }
}

// -x or x, on the integer pipe: the compiler's negation by a condition was an FP64 operation (T170 grid: 61.9 -> 48.3 us)
__device__ __forceinline__ double flip(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? static_cast<int>(0x80000000u) : 0), __double2loint(x));
}
// INV: with the conjugate twiddle
template <bool INV>
__device__ __forceinline__ void fft64_butterfly(int st, int lo, int c, double u, double2 v, const double2 *factors, double &x, double &y) {
  const bool neg = (c != 0) == INV;  // the sign of the sine's term in component c
  if (st < 2) {
    // w = 1, or for the odd butterflies of stage 1 +i (inverse) or -i: i v = (-v.y, v.x)
    const double t = flip((c != 0) != (lo != 0) ? v.y : v.x, lo != 0 && !neg);
    x = u + t;
    y = u - t;
  } else {
    const int h = 1 << st;
    const double2 w = factors[h + lo];
    const bool by_sine = static_cast<unsigned>(4 * lo - h - 1) < static_cast<unsigned>(2 * h - 1), other = (c != 0) != by_sine;
    // component c of w v: cos (a + (+-sin / cos) b) or +-sin (b + (cos / +-sin) a), a = v_c, b the other
    const double t = fma(flip(w.y, neg), other ? v.x : v.y, other ? v.y : v.x), s = flip(w.x, by_sine && neg);
    x = fma(s, t, u);
    y = fma(-s, t, u);
  }
}

}  // namespace lmw
