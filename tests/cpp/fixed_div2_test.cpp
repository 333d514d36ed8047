// div_fixed2 against the IEEE division on the host: the header's device code compiled with the host's correctly
// rounded FMA. Argument: number of divisors. Prints "<divisors> <qualified> <with an exception> <wrong> <not answered>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static double __dmul_rn(double a, double b) { return a * b; }
static long long __double_as_longlong(double x) { long long r; std::memcpy(&r, &x, 8); return r; }
static double __longlong_as_double(long long x) { double r; std::memcpy(&r, &x, 8); return r; }
static int __double2hiint(double x) { return static_cast<int>(__double_as_longlong(x) >> 32); }
static int __double2loint(double x) { return static_cast<int>(__double_as_longlong(x)); }
#include "fixed_div.cuh"

int main(int argc, char **argv) {
  const int want = argc > 1 ? std::atoi(argv[1]) : 1000;
  std::mt19937_64 g(11);
  auto frac = [&] { return 1.0 + std::ldexp(static_cast<double>(g() >> 12), -52); };
  long qualified = 0, exc = 0, wrong = 0, slow = 0;
  for (int n = 0; n < want; n++) {
    double y = std::ldexp(frac(), static_cast<int>(g() % 40) - 20);
    if (n % 3 == 1) y = 1e6 / static_cast<double>(4 + g() % 4000);
    if (n % 3 == 2) y = std::ldexp(static_cast<double>(1 + g() % 4096), static_cast<int>(g() % 8));
    lmw::FixedDiv2 f;
    if (!lmw::fixed_div2_setup(y, f)) continue;
    qualified++;
    exc += f.bad_hi != 0xffffffffu ? 1 : 0;
    for (int k = 0; k < 400; k++) {
      double x;
      if (k == 0) x = 0.0;
      else if (k == 1) x = -0.0;
      else if (k == 2) x = INFINITY;
      else if (k == 3) x = std::nan("");
      else if (k == 4) x = 5e-324;
      else if (k == 5) x = 1.7e308;
      else if (k == 6 && f.bad_hi != 0xffffffffu) x = __longlong_as_double((1023ll << 52) | (static_cast<long long>(f.bad_hi) << 32) | f.bad_lo);
      else if (k & 1) x = frac() * y;                                 // quotients next to a double
      else if (k & 2) x = (frac() + 0x1p-53) * y;                      // quotients next to a midpoint
      else x = std::ldexp(frac(), static_cast<int>(g() % 1700) - 850) * ((g() & 1) ? 1 : -1);
      int ok;
      const double q = lmw::div_fixed2(x, f, ok), r = x / y;
      if (!ok) slow++;
      else if (__double_as_longlong(q) != __double_as_longlong(r)) wrong++;
    }
  }
  std::printf("%d %ld %ld %ld %ld\n", want, qualified, exc, wrong, slow);
  return 0;
}
