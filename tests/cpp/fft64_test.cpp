// The FP64 grid stage's FFT (csrc/fft64.cuh) on the host against long double, beside plain radix-2 butterflies (the product,
// then two sums). Prints, for each length and kind of data, the ratio of the two error norms over the wavenumbers 1 and up
// (forward, then inverse), and the largest error of either relative to the norm of the data, in units of 2^-53.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#define __device__
#define __forceinline__ inline
struct double2 { double x, y; };
static double __hiloint2double(int hi, int lo) { long long b = (static_cast<long long>(hi) << 32) | static_cast<unsigned>(lo); double r; std::memcpy(&r, &b, 8); return r; }
static int __double2hiint(double x) { long long b; std::memcpy(&b, &x, 8); return static_cast<int>(b >> 32); }
static int __double2loint(double x) { long long b; std::memcpy(&b, &x, 8); return static_cast<int>(b); }
using std::fma;
#include "fft64.cuh"

using Row = std::vector<double2>;
static unsigned rev(unsigned k, int logn) { unsigned r = 0; for (int i = 0; i < logn; i++) r |= ((k >> i) & 1u) << (logn - 1 - i); return r; }
template <bool INV> Row ours(const Row &in, int logn, const std::vector<double2> &f) {
  const int n = 1 << logn;
  Row s(n);
  for (int k = 0; k < n; k++) s[rev(k, logn)] = in[k];
  for (int st = 0; st < logn; st++)
    for (int p = 0; p < n / 2; p++) {
      const int h = 1 << st, lo = p & (h - 1), i0 = ((p >> st) << (st + 1)) + lo;
      const double2 u = s[i0], v = s[i0 + h];
      lmw::fft64_butterfly<INV>(st, lo, 0, u.x, v, f.data(), s[i0].x, s[i0 + h].x);
      lmw::fft64_butterfly<INV>(st, lo, 1, u.y, v, f.data(), s[i0].y, s[i0 + h].y);
    }
  return s;
}
template <bool INV> Row plain(const Row &in, int logn) {
  const int n = 1 << logn;
  Row s(n);
  for (int k = 0; k < n; k++) s[rev(k, logn)] = in[k];
  for (int st = 0; st < logn; st++)
    for (int p = 0; p < n / 2; p++) {
      const int h = 1 << st, lo = p & (h - 1), i0 = ((p >> st) << (st + 1)) + lo;
      const long double a = acosl(-1.0L) * lo / h;
      const double wx = static_cast<double>(cosl(a)), wy = static_cast<double>(INV ? sinl(a) : -sinl(a));
      const double2 u = s[i0], v = s[i0 + h], t = {fma(wx, v.x, -(wy * v.y)), fma(wx, v.y, wy * v.x)};
      s[i0] = {u.x + t.x, u.y + t.y};
      s[i0 + h] = {u.x - t.x, u.y - t.y};
    }
  return s;
}
int main() {
  std::mt19937_64 g(3);
  auto uni = [&] { return std::ldexp(static_cast<double>(g() >> 11), -52) - 1; };
  for (int logn = 4; logn <= 9; logn++)
    for (int kind = 0; kind < 3; kind++) {  // values of one size; a mean with small variations; a decaying spectrum
      const int n = 1 << logn, rows = 6144 >> logn;
      std::vector<double2> f(n);
      lmw::fft64_factors(logn, &f[0].x);
      std::vector<long double> c(n), s(n);
      for (int k = 0; k < n; k++) c[k] = cosl(2 * acosl(-1.0L) * k / n), s[k] = sinl(2 * acosl(-1.0L) * k / n);
      double eo[2] = {0, 0}, ep[2] = {0, 0}, most = 0;
      for (int r = 0; r < rows; r++) {
        Row x(n);
        for (int k = 0; k < n; k++) {
          const double z = kind == 1 ? 1e-8 : kind == 2 ? std::pow(1.0 + std::min(k, n - k), -2.0) : 1.0;
          x[k] = {kind == 1 ? 1 + z * uni() : z * uni(), kind == 1 ? 0.7 + z * uni() : z * uni()};
        }
        const Row a[2] = {ours<false>(x, logn, f), ours<true>(x, logn, f)}, b[2] = {plain<false>(x, logn), plain<true>(x, logn)};
        double norm = 0;
        for (int k = 0; k < n; k++) norm += x[k].x * x[k].x + x[k].y * x[k].y;
        for (int k = 0; k < n; k++)
          for (int i = 0; i < 2; i++) {
            long double er = 0, ei = 0;
            for (int j = 0; j < n; j++) {
              const int q = static_cast<int>(static_cast<long>(j) * k % n);
              const long double w = i ? s[q] : -s[q];
              er += c[q] * x[j].x - w * x[j].y;
              ei += c[q] * x[j].y + w * x[j].x;
            }
            auto err = [&](const Row &y) { const double p = static_cast<double>(y[k].x - er), q = static_cast<double>(y[k].y - ei); return p * p + q * q; };
            const double o = err(a[i]);
            if (k || kind == 2) eo[i] += o, ep[i] += err(b[i]);
            most = std::max(most, std::sqrt(o / (norm * n)) * 0x1p53);
          }
      }
      std::printf("%d %d %.4f %.4f %.3f\n", n, kind, std::sqrt(eo[0] / ep[0]), std::sqrt(eo[1] / ep[1]), most);
    }
  return 0;
}
