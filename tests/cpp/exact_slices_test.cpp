// The exact slicing of csrc/exact_slices.cuh on the host: sums of products through the digits, as the tensor cores form them,
// against long double. Argument: number of sums. Prints "<sums> <out of bound> <order past 2^23> <digit out of range> <lost>".
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>
#define __device__
#define __host__
#define __forceinline__ inline
static long long __double_as_longlong(double x) { long long r; std::memcpy(&r, &x, 8); return r; }
static double __longlong_as_double(long long x) { double r; std::memcpy(&r, &x, 8); return r; }
static int __double2hiint(double x) { return static_cast<int>(__double_as_longlong(x) >> 32); }
static double __hiloint2double(int hi, int lo) { return __longlong_as_double((static_cast<long long>(hi) << 32) | static_cast<unsigned>(lo)); }
static unsigned __float_as_uint(float x) { unsigned r; std::memcpy(&r, &x, 4); return r; }
static float __int_as_float(int x) { float r; std::memcpy(&r, &x, 4); return r; }
static int __clzll(long long x) { return x ? __builtin_clzll(static_cast<unsigned long long>(x)) : 64; }
#include "exact_slices.cuh"

int main(int argc, char **argv) {
  const int sums = argc > 1 ? std::atoi(argv[1]) : 1000;
  std::mt19937_64 g(5);
  auto uni = [&] { return std::ldexp(static_cast<double>(g() >> 11), -53); };
  const int scales[] = {0, 0, 0, 900, -880, -930, -1000, -1020, -1060};
  long out = 0, past = 0, bad = 0, lost = 0;
  for (int t = 0; t < sums; t++) {
    // rows of up to 172 values: flat, decaying or rising by up to e^-1 an element, one alone, the ends of the range
    const int K = 1 + static_cast<int>(g() % 172);
    const double da = (g() % 3) * uni(), db = (static_cast<int>(g() % 5) - 2) * 0.5 * uni();
    const int sa = scales[g() % 9], sb = g() % 4 ? 0 : -static_cast<int>(g() % 1000);
    const bool alone = g() % 8 == 0;
    std::vector<double> a(K), b(K);
    int exa = 0, exb = 0;
    for (int k = 0; k < K; k++) {
      a[k] = std::ldexp((2 * uni() - 1) * std::exp(-da * k), sa);
      b[k] = std::ldexp((2 * uni() - 1) * std::exp(db * (k - (db > 0 ? K : 0))), sb);
      if (alone && k) a[k] = 0;
      exa = std::max(exa, lmw::t64_exp(a[k]));
      exb = std::max(exb, lmw::t64_exp(b[k]));
    }
    const int ea = lmw::t64_row(exa), eb = lmw::t64_row(exb);
    int D[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    long double exact = 0;
    for (int k = 0; k < K; k++) {
      unsigned short da8[8], db8[8];
      lmw::t64_digits(lmw::t64_fixed(a[k], ea), da8);
      lmw::t64_digits(lmw::t64_fixed(b[k], eb), db8);
      int va[8], vb[8];
      for (int i = 0; i < 8; i++) {
        va[i] = static_cast<int>(__int_as_float(da8[i] << 16));
        vb[i] = static_cast<int>(__int_as_float(db8[i] << 16));
        if (std::abs(va[i]) > (i ? 64 : 128) || std::abs(vb[i]) > (i ? 64 : 128)) bad++;
      }
      for (int i = 0; i < 8; i++)
        for (int j = 0; i + j < 8; j++) D[i + j] += va[i] * vb[j];
      exact += static_cast<long double>(a[k]) * b[k];
    }
    for (int s = 0; s < 8; s++) past += std::abs(D[s]) >= 1 << 23 ? 1 : 0;
    const lmw::T64Sum r = lmw::t64_sum(D, 1);
    const double got = lmw::t64_value(r.hi, r.lo, ea, eb);
    // Per product: each operand is rounded by 2^-57 of its row's 2^e, and the orders from 8 on leave out at most
    // 7 64^2 2^-70 (1 + 1/128 ...) of 2^(ea + eb); then one rounding of the result
    const long double bound = K * 1.4L * std::ldexp(1.0L, -55 + ea + eb) + std::fabs(exact) * 0x1p-53L + 0x1p-1074L;
    if (!(std::fabs(static_cast<long double>(got) - exact) <= bound)) out++;
    if (got == 0 && std::fabs(exact) > 2 * bound) lost++;
  }
  std::printf("%d %ld %ld %ld %ld\n", sums, out, past, bad, lost);
  return 0;
}
