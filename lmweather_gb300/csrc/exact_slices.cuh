// The integer side of the FP64 Legendre sums on the tensor cores (sphere_tc64.cuh): values of a row scaled by a power of two to
// integers of at most 2^56, their eight digits of seven bits, and the sum of digit products put together and rounded.
#pragma once

namespace lmw {
namespace {

constexpr int T64_DIG = 8;
constexpr int T64_NAN = 100000;  // row exponent of a row that is not finite

// biased exponent of |v| (0 for subnormals and zero)
__device__ __forceinline__ int t64_exp(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }
// row exponent e (every |v| < 2^e) from the largest biased exponent; rows of subnormals and zeros count as those of 2^-1022
__host__ __device__ __forceinline__ int t64_row(int ex) { return ex == 2047 ? T64_NAN : (ex > 1 ? ex : 1) - 1022; }
// v 2^(56 - e) rounded to an integer, by integer operations (|v| < 2^e)
__device__ __forceinline__ long long t64_fixed(double v, int e) {
  const long long bits = __double_as_longlong(v);
  const int be = static_cast<int>((bits >> 52) & 0x7ff), ex = be > 1 ? be : 1, s = 1022 + e - ex;  // right shift of the significand times 8
  if (s > 58 || e == T64_NAN) return 0;
  const long long m8 = ((bits & 0xfffffffffffffll) | (be ? 0x10000000000000ll : 0ll)) << 3;
  const long long x = s > 0 ? (m8 + (1ll << (s - 1))) >> s : m8;
  return bits < 0 ? -x : x;
}
// the eight digits of x, most significant first, as BF16 bits
__device__ __forceinline__ void t64_digits(long long x, unsigned short *out) {
  // digit = ((y + 64) mod 128) - 64, y = (y + 64) / 128: the low four from 28 bits, the others from what they leave
  int y = static_cast<int>(x) & 0xfffffff;
#pragma unroll
  for (int i = T64_DIG - 1; i >= 1; i--) {
    const int u = y + 64;
    y = u >> 7;
    if (i == 4) y += static_cast<int>(x >> 28);  // the carry of the low digits, and the high 29 bits
    out[i] = static_cast<unsigned short>(__float_as_uint(__int_as_float(0x4B400000 | (u & 127)) - 12582976.0f) >> 16);
  }
  out[0] = static_cast<unsigned short>(__float_as_uint(__int_as_float(0x4B400000 + y) - 12582912.0f) >> 16);
}
// sum of the eight orders D[s] (exact integers) times 2^(7 (7 - s)), as high and low parts of value hi 2^28 + lo
struct T64Sum {
  long long hi, lo;
};
__device__ __forceinline__ T64Sum t64_sum(const int *D, int stride) {
  T64Sum r;
  r.hi = ((static_cast<long long>(D[0]) << 21) + (static_cast<long long>(D[stride]) << 14)) + ((static_cast<long long>(D[2 * stride]) << 7) + D[3 * stride]);
  r.lo = ((static_cast<long long>(D[4 * stride]) << 21) + (static_cast<long long>(D[5 * stride]) << 14)) + ((static_cast<long long>(D[6 * stride]) << 7) + D[7 * stride]);
  return r;
}
// (hi 2^28 + lo) 2^(ea + eb - 63) rounded to nearest even, by integer operations (the FP64 pipe would take three times as long);
// |hi|, |lo| < 2^47; ea and eb are the exponents of the operand row and the table row
__device__ __forceinline__ double t64_value(long long hi, long long lo, int ea, int eb) {
  if (ea == T64_NAN) return __longlong_as_double(0x7ff8000000000000ll);
  unsigned long long L = static_cast<unsigned long long>(hi) << 28;
  long long H = hi >> 36;
  L += static_cast<unsigned long long>(lo);
  H += (lo >> 63) + (L < static_cast<unsigned long long>(lo) ? 1 : 0);
  const unsigned long long sign = static_cast<unsigned long long>(H) & 0x8000000000000000ull;
  if (sign) {
    L = 0 - L;
    H = ~H + (L == 0 ? 1 : 0);
  }
  if ((static_cast<unsigned long long>(H) | L) == 0) return 0.0;
  const int p = H ? 127 - __clzll(H) : 63 - __clzll(static_cast<long long>(L));  // the leading bit
  unsigned long long m;
  if (p <= 52) {
    m = L << (52 - p);
  } else {
    const int sh = p - 52;  // at most 24: |hi 2^28 + lo| < 2^76
    m = (static_cast<unsigned long long>(H) << (64 - sh)) | (L >> sh);
    const unsigned long long rem = L & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    m += rem > half || (rem == half && (m & 1)) ? 1 : 0;
  }
  const int x = p + 1023 + ea + eb - 63;  // biased exponent
  if (x >= 1 && x <= 2045) return __longlong_as_double(static_cast<long long>(sign | ((static_cast<unsigned long long>(x - 1) << 52) + m)));
  // the ends of the range: scale in two steps (below 2^-1200 the value, less than 2^77 before, is less than the least subnormal's half)
  const double v = __longlong_as_double(static_cast<long long>(sign | ((static_cast<unsigned long long>(p + 1022) << 52) + m)));
  const int e = ea + eb - 63 > -1200 ? ea + eb - 63 : -1200, e1 = e / 2;
  return v * __hiloint2double((e1 + 1023) << 20, 0) * __hiloint2double((e - e1 + 1023) << 20, 0);
}

}  // namespace
}  // namespace lmw
