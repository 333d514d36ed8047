// FP64 Legendre sums on the tensor cores by exact slicing (included by sphere.cu), truncations up to 170.
//
// GB300's FP64 pipe does about 0.5e12 multiply-adds a second, its BF16 tensor cores a thousand times that. The sums of a
// wavenumber m are therefore formed from integers (the scheme of K. Ozaki, T. Ogita, S. Oishi and S. M. Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix multiplication and its applications",
// Numerical Algorithms 59, 2012): every operand row is scaled by a power of two to integers of at most 2^56 and cut into
// eight digits of seven bits (d_0 up to 128, the others -64..63), which BF16 holds exactly. The products of two digits
// summed over a row of at most 172 coefficients or 128 latitudes, for all digit pairs (i, j) of one order s = i + j, stay
// below 2^23, so the FP32 accumulators of tcgen05 hold them exactly. The eight orders s = 0..7 are then added as 64-bit
// integers and rounded once: a sum of K products of rows below 2^ea and 2^eb is within 1.4 K 2^-55 2^(ea + eb) and one rounding
// of the exact one (each operand rounded by 2^-57 of its row, the orders from 8 on left out), and depends neither on the
// order of summation nor on how members are batched. A row with an infinity or NaN gives NaN.
// That is a bound by norm, by the largest coefficient and the largest table value of a row. Of a wavenumber's largest value the
// error is 0.04e-15 to 0.9e-15 (T170, spectra from flat to n^-3; plain FP64 sums 0.06e-15 to 1.7e-15). A value far below it, as a
// high wavenumber has towards the poles where its large coefficients meet table values far below the row's largest,
// keeps fewer digits than a plain sum would give it, or none. A stage adds such values to those of all other
// wavenumbers in an FFT, whose rounding is by norm as well, and its sums over latitudes are dominated by the others: against
// extended precision the error of each wavenumber after two steps is 0.86 to 1.02 of that with plain sums and radix-2 FFTs for
// delta and Phi, 0.56 to 1.02 for zeta (T21 to T170; a small perturbation of a zonal flow, steep and flat spectra). What is
// handed out as a grid takes plain sums (SphereEngine::synth_grids).
//
// All orders of one table digit j come from one MMA: A holds digit i of its rows in row block i, under seven blocks of
// zeros, and for table digit j the MMA starts j blocks higher, which puts digit i into row block i + j of the accumulator.
//
// Sums use P_n^m alone, n = m..T+1. With (1 - mu^2) dP_n/dmu = -n eps_{n+1} P_{n+1} + (n+1) eps_n P_{n-1}
// (cpp/sphere.cpp:91-94) the derivative terms of cpp/sphere.cpp:192-202 become spectral coefficients of U and V, and
// those of cpp/sphere.cpp:364-371 combinations of the sums at n - 1 and n + 1: four sums instead of six, five instead of
// seven, and one table.
//
// tc64_syn   one CTA per (m, up to 64 latitude pairs, one or two members): U, V, zeta, Phi coefficients -> digits in shared
//            memory (rows: four complex values per member) -> even and odd n - m in two accumulators -> Fourier
//            coefficients of both mirror latitudes.
// tc64_ana   one CTA per (m, member): folded grid values -> digits (rows: five complex values) -> sums of both
//            parities -> tendencies, RK4 update, filter.
// The table digits are streamed by bulk copies, sixteen K columns of all eight digits a stage, and start before the
// kernel waits for its predecessor.
#pragma once
#include "exact_slices.cuh"
#include "tc_common.cuh"

namespace lmw {

struct Tc64Plan {
  int nh16 = 16, lrows = 16, nsl = 1, nhk = 16;  // padded latitude pairs, per slice, slices; K of the analysis
  int ns = 3, nsa = 3;                           // table chunks in flight: synthesis, analysis
  int nbt = 1, ntiles = 1;                               // members per synthesis tile
  int kc_max = 1, ra_max = 16;
  bool wide = false;  // analysis CTAs of 512 threads
  size_t smem_ana = 0;
  size_t smem_syn(int blocks) const;  // row blocks of eight rows (members; two with the tracer)
  DevBuf<__nv_bfloat16> tS, tA;
  DevBuf<int> ke16, kc, ra16;    // synthesis: padded even columns, K chunks of 16; analysis: padded rows of (m, parity)
  DevBuf<long> oS, oA;           // table offsets (elements)
  DevBuf<int> eS, eA;            // row exponents: [m][nh16], [tri + m + n - m] (n to T+1)
  DevBuf<double> cf;             // per (m, n), n to T+1, five coefficients (see Tc64Dev)
  HostBuf<int> err;              // written by the device when a bounded wait ran out
};

struct Tc64Dev {
  int nh16, lrows, nsl, nhk, ns, nsa, nbt, ntiles, ra_max, ext;  // ext: coefficients with n to T+1
  const __nv_bfloat16 *tS, *tA;
  const int *ke16, *kc, *ra16, *eS, *eA;
  const long *oS, *oA;
  const double *cf;  // [5][ext]: a m / (n (n+1)), a eps_n / n, a eps_{n+1} / (n+1), n eps_{n+1}, (n+1) eps_n
  int *err;
};

namespace {

constexpr int T64_THREADS = 256, T64_STAGES = 8;  // T64_STAGES: most chunks in flight
// A operand: core matrices 128 bytes apart along K and 256 between 8-row groups. The digits' stores meet four to a bank;
// with 16 spare bytes between core matrices they do not, which changed no time (T42 x 16, T170: within 2 %)
constexpr int T64_LBO = 128, T64_SBO = 256;

__device__ __forceinline__ uint64_t t64_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(lbo >> 4) << 16) | (static_cast<uint64_t>(sbo >> 4) << 32) |
         (static_cast<uint64_t>(1) << 46);
}

// ------------------------------------------------------------------------------------------------ tables
// P_n^m at latitude pair jh, n to T+1 (P1: the row n = T+1)
__device__ __forceinline__ double t64_p(const SphDev &d, const double *P1, int m, int n, int jh) {
  return n <= d.N ? d.Ps[static_cast<size_t>(d.tri[m] + n - m) * d.nh + jh] : P1[static_cast<size_t>(m) * d.nh + jh];
}
// digits of the synthesis table: [slice][chunk][digit][lrows][16] in core matrices, rows latitudes, columns even n - m then
// odd; grid M, thread: latitude
__global__ void tc64_build_syn(SphDev d, Tc64Dev z, const double *__restrict__ P1, __nv_bfloat16 *__restrict__ tS, int *__restrict__ eS) {
  const int m = blockIdx.x, kc = z.kc[m], ke16 = z.ke16[m];
  for (int jh = threadIdx.x; jh < z.nh16; jh += blockDim.x) {
    int ex = 0;
    for (int n = m; n <= d.N + 1 && jh < d.nh; n++) ex = max(ex, t64_exp(t64_p(d, P1, m, n, jh)));
    const int e = t64_row(ex), sl = jh / z.lrows, r = jh % z.lrows;
    eS[m * z.nh16 + jh] = e;
    for (int k = 0; k < kc * 16; k++) {
      const int n = k < ke16 ? m + 2 * k : m + 1 + 2 * (k - ke16);
      unsigned short dg[T64_DIG];
      t64_digits(jh < d.nh && n <= d.N + 1 ? t64_fixed(t64_p(d, P1, m, n, jh), e) : 0, dg);
      unsigned short *o = reinterpret_cast<unsigned short *>(tS) + z.oS[m] + (static_cast<long>(sl) * kc + k / 16) * T64_DIG * z.lrows * 16;
      for (int i = 0; i < T64_DIG; i++) o[(i * z.lrows + (r & ~7)) * 16 + ((k & 15) >> 3) * 64 + (r & 7) * 8 + (k & 7)] = dg[i];
    }
  }
}
// digits of the analysis table of (m, parity): [chunk][digit][ra16][16], rows n = m + parity + 2 r, columns latitudes; grid
// (M, 2), one warp per row
__global__ void tc64_build_ana(SphDev d, Tc64Dev z, const double *__restrict__ P1, __nv_bfloat16 *__restrict__ tA, int *__restrict__ eA) {
  const int m = blockIdx.x, p = blockIdx.y, ra = z.ra16[2 * m + p], lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < ra; r += blockDim.x >> 5) {
    const int n = m + p + 2 * r;
    int ex = 0;
    if (n <= d.N + 1)
      for (int jh = lane; jh < d.nh; jh += 32) ex = max(ex, t64_exp(t64_p(d, P1, m, n, jh)));
    ex = __reduce_max_sync(0xffffffffu, ex);
    const int e = t64_row(ex);
    if (lane == 0 && n <= d.N + 1) eA[d.tri[m] + m + n - m] = e;
    for (int k = lane; k < z.nhk; k += 32) {
      unsigned short dg[T64_DIG];
      t64_digits(k < d.nh && n <= d.N + 1 ? t64_fixed(t64_p(d, P1, m, n, k), e) : 0, dg);
      unsigned short *o = reinterpret_cast<unsigned short *>(tA) + z.oA[2 * m + p] + static_cast<long>(k / 16) * T64_DIG * ra * 16;
      for (int i = 0; i < T64_DIG; i++) o[(i * ra + (r & ~7)) * 16 + ((k & 15) >> 3) * 64 + (r & 7) * 8 + (k & 7)] = dg[i];
    }
  }
}

// ------------------------------------------------------------------------------------------------ shared pieces
struct T64Bars {
  uint64_t full[T64_STAGES], empty[T64_STAGES], done;
  uint32_t tslot;
  int fail, issued, consumed;
};
// tensor memory (warp 0) and barriers
__device__ __forceinline__ void t64_setup(T64Bars &b, int ns, uint32_t ncols) {
  if (threadIdx.x < 32) tc::tmem_alloc(tc::su32(&b.tslot), ncols);
  if (threadIdx.x == 0) {
    for (int s = 0; s < ns; s++) {
      tc::bar_init(tc::su32(&b.full[s]), 1);
      tc::bar_init(tc::su32(&b.empty[s]), 1);
    }
    tc::bar_init(tc::su32(&b.done), 1);
    tc::bar_init_fence();
    b.fail = b.issued = b.consumed = 0;
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
}
__device__ __forceinline__ void t64_failed(T64Bars &b, int *err, int code) {
  b.fail = 1;
  *reinterpret_cast<volatile int *>(err) = code;
  __threadfence_system();
}
// producer step: chunk it (bytes from src) into stage it % ns
__device__ __forceinline__ bool t64_copy(T64Bars &b, uint8_t *stages, int stage_bytes, int ns, int it, const void *src, uint32_t bytes, int *err) {
  const int st = it % ns;
  if (it >= ns && !tc::wait(tc::su32(&b.empty[st]), ((it / ns) - 1) & 1)) {
    t64_failed(b, err, 11);
    return false;
  }
  tc::expect_tx(tc::su32(&b.full[st]), bytes);
  tc::bulk_g2s(tc::su32(stages + static_cast<size_t>(st) * stage_bytes), src, bytes, tc::su32(&b.full[st]));
  b.issued = it + 1;
  return true;
}
// MMA step, by a whole warp (`leader`: its issuing lane): the eight table digits of stage it % ns (rows: N) against the A
// block at `a` (its first real row group 7 gpo groups further down, gpo groups per digit), accumulated at `acc`
__device__ __forceinline__ bool t64_mma(T64Bars &b, uint32_t stages, int stage_bytes, int ns, int it, int N, uint32_t a, int gpo, uint32_t acc, bool first,
                                        bool leader, int *err) {
  const int st = it % ns;
  if (!tc::wait_warp(tc::su32(&b.full[st]), (it / ns) & 1)) {
    t64_failed(b, err, 12);
    return false;
  }
  tc::fence_after();
  const uint64_t ad = t64_desc(a + 7 * gpo * T64_SBO, T64_LBO, T64_SBO), bd = t64_desc(stages + st * stage_bytes, 128, 256);
  const uint32_t idesc = tc::idesc_m128(N);
  b.consumed = it + 1;
#pragma unroll
  for (int j = 0; j < T64_DIG; j++)
    tc::mma(leader, acc, ad - static_cast<uint64_t>(j * gpo * (T64_SBO / 16)), bd + static_cast<uint64_t>(j * N * 2), idesc, first && j == 0 ? 0u : 1u);
  tc::commit(leader, tc::su32(&b.empty[st]));
  return true;
}
// after the roles have met: wait for every MMA; after a failure a bounded wait for what is in flight. True when all is well
__device__ __forceinline__ bool t64_finish(T64Bars &b, int ns, int *err) {
  __syncthreads();
  if (threadIdx.x == 0) {
    if (!b.fail) {
      if (!tc::wait(tc::su32(&b.done), 0)) t64_failed(b, err, 13);
    } else {
      tc::wait_for(tc::su32(&b.done), 0, 200000000ull);
      for (int it = b.consumed; it < b.issued; it++) tc::wait_for(tc::su32(&b.full[it % ns]), (it / ns) & 1, 200000000ull);
    }
  }
  __syncthreads();
  tc::fence_after();
  return b.fail == 0;
}
__device__ __forceinline__ void t64_teardown(T64Bars &b, uint32_t ncols) {
  tc::fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tc::tmem_free(b.tslot, ncols);
}
// 32 (or the first w = 16) accumulator columns of this thread's row as integers into dst
__device__ __forceinline__ void t64_unload(uint32_t taddr, int w, int *dst, bool keep) {
  float v[32];
  if (w > 16) {
    tc::ld32(taddr, v);
  } else {
    tc::ld8(taddr, v);
    tc::ld8(taddr + 8, v + 8);
  }
  if (!keep) return;
#pragma unroll
  for (int i = 0; i < 32; i++)
    if (i < w) dst[i] = __float2int_rn(v[i]);
}

// ------------------------------------------------------------------------------------------------ synthesis
// grid: (slices x tiles, M). F = 4: U, V, zeta, Phi of x [B][3][ntri] into four [B][nlat][4][M], nbt members a tile; F = 6: with
// the tracer's q of qin [B][ntri] and delta of x into fourq [B][nlat][2][M], one member a tile, whose second row block is q
// and delta.
// T170, one member: 82.0 -> 18.2 us (FP64 pipe before); T42 x 16: 50.4 -> 10.3; T42, one member: 10.3 -> 6.5.
template <int F>
__global__ void __launch_bounds__(T64_THREADS, 2) tc64_syn(SphDev d, Tc64Dev z, const double2 *__restrict__ x, const double2 *__restrict__ qin,
                                                           double2 *__restrict__ four, double2 *__restrict__ fourq, int B) {
  extern __shared__ __align__(1024) uint8_t t64_sm[];
  __shared__ __align__(8) T64Bars bars;
  constexpr int RF = 4;  // complex values of a row block
  __shared__ int rowexp[2][RF];
  const int tid = threadIdx.x, m = blockIdx.y, sl = blockIdx.x % z.nsl, tile = blockIdx.x / z.nsl;
  // nbt row blocks: members, or the flow and the tracer of one
  const int L = z.lrows, kc = z.kc[m], ke16 = z.ke16[m], nbt = F == 6 ? 2 : z.nbt, mt = F == 6 ? 2 : min(nbt, B - tile * nbt), groups = 15 * nbt;
  const int stage_bytes = T64_DIG * L * 32, ablk = groups * T64_SBO;
  uint8_t *stages = t64_sm;
  uint8_t *A = t64_sm + max(z.ns * stage_bytes, static_cast<int>(2 * 64 * nbt * (min(L, 32) + 1) * sizeof(int)));
  const uint32_t ncols = max(32, 2 * L);
  t64_setup(bars, z.ns, ncols);
  const __nv_bfloat16 *src = z.tS + z.oS[m] + static_cast<long>(sl) * kc * T64_DIG * L * 16;
  int copied = 0;
  if (tid == 0)
    for (; copied < min(kc, z.ns); copied++) t64_copy(bars, stages, stage_bytes, z.ns, copied, src + static_cast<long>(copied) * T64_DIG * L * 16, stage_bytes, z.err);
  // the zero blocks above the digits
  for (int e = tid; e < kc * 7 * nbt * (T64_SBO / 16); e += T64_THREADS) {
    const int blk = e / (7 * nbt * (T64_SBO / 16)), o = e % (7 * nbt * (T64_SBO / 16));
    *reinterpret_cast<uint4 *>(A + blk * ablk + o * 16) = make_uint4(0, 0, 0, 0);
  }
  if (tid < 2 * RF) rowexp[tid / RF][tid % RF] = 0;
  __syncthreads();
  pdl_wait(x, qin);
  // items: a complex value f of row block ml at column k, n = m + 2 k or m + 1 + 2 (k - ke16). Columns are padded to 16, so
  // that a half warp has one (ml, f)
  const int cols = kc * 16, total = (F == 6 ? 6 : 4 * mt) * cols, base = d.tri[m] - m;
  constexpr int IT = ((F == 6 ? 6 : 8) * 192 + T64_THREADS - 1) / T64_THREADS;
  auto where = [&](int e, int &ml, int &f, int &k) {
    const int v = e / cols;
    k = e - v * cols;
    ml = v >> 2;
    f = v & 3;
  };
  double v[IT][2];
#pragma unroll
  for (int r = 0; r < IT; r++) {
    const int e = tid + r * T64_THREADS;
    if (e >= total) break;
    int ml, f, k;
    where(e, ml, f, k);
    const int n = k < ke16 ? m + 2 * k : m + 1 + 2 * (k - ke16);
    const int b = F == 6 ? tile : tile * nbt + ml;
    const double2 *xz = x + static_cast<size_t>(b) * 3 * d.ntri + base, *xd = xz + d.ntri, *xf = xd + d.ntri;
    const double2 zero = make_double2(0.0, 0.0);
    const bool flow = F == 4 || ml == 0;
    const double2 *ce = flow ? (f == 0 ? xd : f == 3 ? xf : xz) : f == 0 ? qin + static_cast<size_t>(b) * d.ntri + base : xd;
    const double2 c = n <= d.N ? ce[n] : zero;
    v[r][0] = c.x;
    v[r][1] = c.y;
    if (flow && f < 2) {
      // U_n = -a [i m delta_n / (n (n+1)) + eps_n zeta_{n-1} / n - eps_{n+1} zeta_{n+1} / (n+1)], V_n the same with zeta_n,
      // -delta_{n-1}, -delta_{n+1}; the (0, 0) coefficients have no wind
      const double2 *nb = f == 0 ? xz : xd;
      const bool live = n <= d.N + 1;
      const double *cf = z.cf + d.tri[m] + (live ? n : m);  // ext index of (m, n): tri[m] + m + n - m
      const double w0 = live ? cf[0] : 0.0, w1 = live ? cf[z.ext] : 0.0, w2 = live ? cf[2 * z.ext] : 0.0;
      const double2 l = n > m && n > 1 && n <= d.N + 1 ? nb[n - 1] : zero, u = n < d.N ? nb[n + 1] : zero;
      if (f == 0) {
        v[r][0] = fma(w0, c.y, fma(w2, u.x, -(w1 * l.x)));
        v[r][1] = fma(-w0, c.x, fma(w2, u.y, -(w1 * l.y)));
      } else {
        v[r][0] = fma(w0, c.y, fma(w1, l.x, -(w2 * u.x)));
        v[r][1] = fma(-w0, c.x, fma(w1, l.y, -(w2 * u.y)));
      }
    }
    const int ex = __reduce_max_sync(0xffffu << (tid & 16), max(t64_exp(v[r][0]), t64_exp(v[r][1])));
    if ((tid & 15) == 0) atomicMax(&rowexp[ml][f], ex);
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < IT; r++) {
    const int e = tid + r * T64_THREADS;
    if (e >= total) break;
    int ml, f, k;
    where(e, ml, f, k);
    uint8_t *o = A + (k >> 4) * ablk + (7 * nbt + ml) * T64_SBO + ((k & 15) >> 3) * T64_LBO + (k & 7) * 2 + f * 32;
    const int er = t64_row(rowexp[ml][f]);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      unsigned short dg[T64_DIG];
      t64_digits(t64_fixed(v[r][q], er), dg);
#pragma unroll
      for (int i = 0; i < T64_DIG; i++) *reinterpret_cast<unsigned short *>(o + i * nbt * T64_SBO + q * 16) = dg[i];
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const uint32_t tmem = bars.tslot;
  const int role = tc::uniform(tid >> 5);
  if (tid == 0) {
    for (; copied < kc; copied++)
      if (!t64_copy(bars, stages, stage_bytes, z.ns, copied, src + static_cast<long>(copied) * T64_DIG * L * 16, stage_bytes, z.err)) break;
  } else if (role == 1) {
    const int even = ke16 / 16;
    const uint32_t s0 = tc::su32(stages), a0 = tc::su32(A), t0 = tc::uniform(tmem);
    const bool leader = tc::elect_one();
    for (int c = 0; c < kc; c++)
      if (!t64_mma(bars, s0, stage_bytes, z.ns, c, L, a0 + c * ablk, nbt, t0 + (c < even ? 0 : L), c == 0 || c == even, leader, z.err)) break;
    tc::commit(leader, tc::su32(&bars.done));
  }
  const bool ok = t64_finish(bars, z.ns, z.err);
  pdl_trigger();
  const int warp = tid >> 5, lane = tid & 31, quarter = warp & 3, row = quarter * 32 + lane, rows = 64 * nbt;
  int *red = reinterpret_cast<int *>(t64_sm);  // [2][rows][w + 1]: even, odd
  const int w = min(L, 32), ld = w + 1;
  for (int cb = 0; ok && cb < L; cb += 32) {
    if (quarter * 32 < rows)
      t64_unload(tmem + (warp < 4 ? 0 : L) + cb + (static_cast<uint32_t>(quarter * 32) << 16), w, red + ((warp < 4 ? 0 : rows) + row) * ld, row < rows);
    __syncthreads();
    for (int e = tid; e < (F == 6 ? 6 : 4 * mt) * w; e += T64_THREADS) {
      const int i = e % w, v = e / w, f = v & 3, ml = v >> 2, jh = sl * L + cb + i;
      if (jh >= d.nh) continue;
      const int ea = t64_row(rowexp[ml][f]), eb = z.eS[m * z.nh16 + jh];
      double so[2], no[2];
#pragma unroll
      for (int ri = 0; ri < 2; ri++) {
        const int r0 = ml * 8 + 2 * f + ri;
        const T64Sum ev = t64_sum(red + r0 * ld + i, 8 * nbt * ld), od = t64_sum(red + (rows + r0) * ld + i, 8 * nbt * ld);
        so[ri] = t64_value(ev.hi + od.hi, ev.lo + od.lo, ea, eb);
        no[ri] = t64_value(ev.hi - od.hi, ev.lo - od.lo, ea, eb);
      }
      const bool trc = F == 6 && ml == 1;
      const size_t bo = static_cast<size_t>(F == 6 ? tile : tile * nbt + ml) * d.nlat;
      const int W = trc ? 2 : 4;
      double2 *o = (trc ? fourq : four) + f * d.M + m;
      o[(bo + jh) * W * d.M] = make_double2(so[0], so[1]);
      o[(bo + d.nlat - 1 - jh) * W * d.M] = make_double2(no[0], no[1]);
    }
    __syncthreads();
  }
  t64_teardown(bars, ncols);
}

// ------------------------------------------------------------------------------------------------ analysis + RK4
// grid: (B, M). SLOTS = 5: the flow (fold [B][nh][5][2][M]; x0, xs, acc [B][3][ntri]); SLOTS = 8: with the tracer (foldq
// [B][nh][3][2][M]: U q, V q, q delta; q0, qs, qacc [B][ntri]).
// T170, one member: 71.7 -> 29.8 us; T42 x 16: 45.1 -> 26.2; T42, one member: 8.2 -> 7.5.
template <int SLOTS, int NT>
__global__ void __launch_bounds__(NT, 1) tc64_ana(SphDev d, Tc64Dev z, const double2 *__restrict__ fold, StageArgs sa, double2 *__restrict__ x0,
                                                           double2 *__restrict__ xs, double2 *__restrict__ acc, const double2 *__restrict__ foldq,
                                                           double2 *__restrict__ q0, double2 *__restrict__ qs, double2 *__restrict__ qacc) {
  constexpr int Q = 2 * SLOTS, FIELDS = SLOTS == 8 ? 4 : 3, GPO = 2;  // GPO: row groups per digit
  extern __shared__ __align__(1024) uint8_t t64_sm[];
  __shared__ __align__(8) T64Bars bars;
  __shared__ int rowexp[2][Q];
  const int tid = threadIdx.x, m = blockIdx.y, b = blockIdx.x;
  const int kc = z.nhk / 16, ra0 = z.ra16[2 * m], ra1 = z.ra16[2 * m + 1], stage_bytes = T64_DIG * z.ra_max * 32, ablk = 15 * GPO * T64_SBO;
  uint8_t *stages = t64_sm, *A = t64_sm + z.nsa * stage_bytes;
  uint32_t ncols = 32;
  while (ncols < static_cast<uint32_t>(ra0 + ra1)) ncols <<= 1;
  t64_setup(bars, z.nsa, ncols);
  // chunks: parity 0's kc, then parity 1's
  auto chunk = [&](int it) { return z.tA + z.oA[2 * m + (it < kc ? 0 : 1)] + static_cast<long>(it < kc ? it : it - kc) * T64_DIG * (it < kc ? ra0 : ra1) * 16; };
  auto bytes = [&](int it) { return static_cast<uint32_t>(T64_DIG * (it < kc ? ra0 : ra1) * 32); };
  int copied = 0;
  if (tid == 0)
    for (; copied < min(2 * kc, z.nsa); copied++) t64_copy(bars, stages, stage_bytes, z.nsa, copied, chunk(copied), bytes(copied), z.err);
  for (int e = tid; e < 2 * kc * 7 * GPO * (T64_SBO / 16); e += NT) {
    const int blk = e / (7 * GPO * (T64_SBO / 16)), o = e % (7 * GPO * (T64_SBO / 16));
    *reinterpret_cast<uint4 *>(A + blk * ablk + o * 16) = make_uint4(0, 0, 0, 0);
  }
  if (tid < 2 * Q) rowexp[tid / Q][tid % Q] = 0;
  __syncthreads();
  pdl_wait(fold, foldq, x0, xs, acc, q0, qs, qacc);
  // items: slot s of latitude pair jh at parity p of the fold; pairs are padded to 16, so that a half warp has one (s, p)
  const int items = SLOTS * 2 * z.nhk;
  constexpr int IT = (SLOTS * 256 + NT - 1) / NT;
  auto where = [&](int e, int &s, int &p, int &jh) {
    jh = e & (z.nhk - 1);  // a power of two
    p = e / z.nhk & 1;
    s = e / z.nhk >> 1;
  };
  double v[IT][2];
#pragma unroll
  for (int r = 0; r < IT; r++) {
    const int e = tid + r * NT;
    int s, p, jh;
    where(e, s, p, jh);
    v[r][0] = v[r][1] = 0;
    if (e < items && jh < d.nh) {
      const double2 *src = s < 5 ? fold + ((static_cast<size_t>(b) * d.nh + jh) * 5 + s) * 2 * d.M : foldq + ((static_cast<size_t>(b) * d.nh + jh) * 3 + s - 5) * 2 * d.M;
      const double2 g = src[p * d.M + m];
      v[r][0] = g.x;
      v[r][1] = g.y;
    }
  }
#pragma unroll
  for (int r = 0; r < IT; r++) {
    const int e = tid + r * NT;
    if (e >= items) break;
    int s, p, jh;
    where(e, s, p, jh);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int ex = __reduce_max_sync(0xffffu << (tid & 16), t64_exp(v[r][q]));
      if ((tid & 15) == 0) atomicMax(&rowexp[p][2 * s + q], ex);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < IT; r++) {
    const int e = tid + r * NT;
    if (e >= items) break;
    int s, p, jh;
    where(e, s, p, jh);
    uint8_t *o = A + (p * kc + (jh >> 4)) * ablk + 7 * GPO * T64_SBO + ((jh & 15) >> 3) * T64_LBO + (jh & 7) * 2 + (s >> 2) * T64_SBO + (s & 3) * 32;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      unsigned short dg[T64_DIG];
      t64_digits(t64_fixed(v[r][q], t64_row(rowexp[p][2 * s + q])), dg);
#pragma unroll
      for (int i = 0; i < T64_DIG; i++) *reinterpret_cast<unsigned short *>(o + i * GPO * T64_SBO + q * 16) = dg[i];
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const uint32_t tmem = bars.tslot;
  const int role = tc::uniform(tid >> 5);
  if (tid == 0) {
    for (; copied < 2 * kc; copied++)
      if (!t64_copy(bars, stages, stage_bytes, z.nsa, copied, chunk(copied), bytes(copied), z.err)) break;
  } else if (role == 1) {
    const uint32_t s0 = tc::su32(stages), a0 = tc::su32(A), t0 = tc::uniform(tmem);
    const bool leader = tc::elect_one();
    for (int it = 0; it < 2 * kc; it++)
      if (!t64_mma(bars, s0, stage_bytes, z.nsa, it, it < kc ? ra0 : ra1, a0 + it * ablk, GPO, t0 + (it < kc ? 0 : ra0), it == 0 || it == kc, leader, z.err)) break;
    tc::commit(leader, tc::su32(&bars.done));
  }
  // item e of the update: field e / cnt, n = m + e % cnt. What it reads is loaded while the MMAs run
  const int cnt = d.N + 1 - m;
  // field f of item i: the flow's three, then the tracer
  auto place = [&](int f, int i) { return (f < 3 ? static_cast<size_t>(b) * 3 + f : static_cast<size_t>(b)) * d.ntri + d.tri[m] + i; };
  constexpr int ITEMS = (FIELDS * 171 + NT - 1) / NT;
  double2 xv[ITEMS], av[ITEMS];
  double w3[ITEMS], w4[ITEMS], lap[ITEMS], fac[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    const int e = tid + r * NT, f = e / cnt, i = e - f * cnt;
    xv[r] = av[r] = make_double2(0.0, 0.0);
    w3[r] = w4[r] = lap[r] = fac[r] = 0;
    if (f < FIELDS) {
      const size_t o = place(f, i);
      xv[r] = (f < 3 ? x0 : q0)[o];
      if (sa.stage > 0) av[r] = (f < 3 ? acc : qacc)[o];
      w3[r] = z.cf[3 * z.ext + d.tri[m] + m + i];
      w4[r] = z.cf[4 * z.ext + d.tri[m] + m + i];
      if (f == 1) lap[r] = d.lapl[m + i];
      if (sa.stage == 3) fac[r] = sa.filt[(f >= 2 ? 1 : 0) * d.M + m + i];
    }
  }
  const bool ok = t64_finish(bars, z.nsa, z.err);
  pdl_trigger();
  // sums S[q][n - m], n to T+1
  const int warp = tid >> 5, lane = tid & 31, quarter = warp & 3, row = quarter * 32 + lane, next = d.N + 2 - m;
  constexpr int ROWS = 64 * GPO, LD = 33, NB = NT / 128;  // NB column blocks of 32 at once
  int *red = reinterpret_cast<int *>(t64_sm);                                   // [NB][ROWS][LD]
  double *S = reinterpret_cast<double *>(t64_sm + ((NB * ROWS * LD * sizeof(int) + 15) & ~15u));  // [Q][next + 1]
  const int sld = next + 1, total = ra0 + ra1;
  for (int cb = 0; ok && cb < total; cb += 32 * NB) {
    const int c0 = cb + (warp >> 2) * 32, w = total - c0 >= 32 ? 32 : 16;
    if (quarter * 32 < ROWS && c0 < total)
      t64_unload(tmem + c0 + (static_cast<uint32_t>(quarter * 32) << 16), w, red + ((warp >> 2) * ROWS + row) * LD, true);
    __syncthreads();
    for (int e = tid; e < Q * 32 * NB; e += NT) {
      const int i = e & (32 * NB - 1), q = e / (32 * NB), c = cb + i, pp = c < ra0 ? 0 : 1, r = pp ? c - ra0 : c, nn = m + pp + 2 * r;
      if (c >= total || nn > d.N + 1) continue;
      const T64Sum t = t64_sum(red + ((i >> 5) * ROWS + (q >> 3) * 8 + (q & 7)) * LD + (i & 31), 8 * GPO * LD);
      S[q * sld + nn - m] = t64_value(t.hi, t.lo, t64_row(rowexp[pp][q]), z.eA[d.tri[m] + nn]);
    }
    __syncthreads();
  }
  if (ok) {
    const double mm = static_cast<double>(m);
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
      const int e = tid + r * NT, f = e / cnt, i = e - f * cnt, q = d.tri[m] + i;
      if (f >= FIELDS) continue;
      auto at = [&](int s) { return make_double2(S[2 * s * sld + i], S[(2 * s + 1) * sld + i]); };
      // the H sum: -n eps_{n+1} S(n+1) + (n+1) eps_n S(n-1)
      auto deriv = [&](int s) {
        const double2 u = make_double2(S[2 * s * sld + i + 1], S[(2 * s + 1) * sld + i + 1]);
        const double2 l = i > 0 ? make_double2(S[2 * s * sld + i - 1], S[(2 * s + 1) * sld + i - 1]) : make_double2(0.0, 0.0);
        return make_double2(fma(w4[r], l.x, -(w3[r] * u.x)), fma(w4[r], l.y, -(w3[r] * u.y)));
      };
      double2 k;
      if (f < 3) {
        // cpp/sphere.cpp:380-383: dz = -D(A,B), dd = D(B,-A) + n(n+1)/a^2 (Phi + E), df = -D(U Phi, V Phi)
        // slots: A, B, U Phi, V Phi, Phi + E; the zonal terms take A, B, U Phi, the others B, A, V Phi
        const double2 dv = deriv(f == 0 ? 1 : f == 1 ? 0 : 3), iv = imul(at(f), mm);
        k = f == 1 ? cadd(cadd(iv, dv), cscale(at(4), lap[r])) : csub(dv, iv);
        if (q == 0 || sa.zero) k = make_double2(0.0, 0.0);  // cpp/sphere.cpp:387-389
      } else {
        k = cadd(at(7), csub(deriv(6), imul(at(5), mm)));  // dq = A(q delta) - D(U q, V q), cpp/sphere.cpp:250-263
      }
      const size_t o = place(f, i);
      if (sa.stage < 3) {
        (f < 3 ? acc : qacc)[o] = sa.stage == 0 ? k : make_double2(fma(2.0, k.x, av[r].x), fma(2.0, k.y, av[r].y));
        (f < 3 ? xs : qs)[o] = make_double2(fma(sa.c, k.x, xv[r].x), fma(sa.c, k.y, xv[r].y));
      } else {
        // cpp/sphere.cpp:428-434: x += dt/6 (k1 + 2k2 + 2k3 + k4), then the del^4 filter (the tracer: Phi's)
        const double2 val = make_double2(fma(sa.c, av[r].x + k.x, xv[r].x), fma(sa.c, av[r].y + k.y, xv[r].y));
        (f < 3 ? x0 : q0)[o] = q == 0 ? val : cscale(val, fac[r]);
      }
    }
  }
  t64_teardown(bars, ncols);
}

}  // namespace

inline Tc64Dev tc64_dev(const Tc64Plan &p, int ext) {
  return Tc64Dev{p.nh16, p.lrows, p.nsl, p.nhk, p.ns, p.nsa, p.nbt, p.ntiles, p.ra_max, ext, p.tS.p, p.tA.p, p.ke16.p, p.kc.p, p.ra16.p, p.eS.p, p.eA.p, p.oS.p, p.oA.p, p.cf.p, p.err.p};
}

// an M = 128 MMA reads sixteen row groups from its A block: with one row block of eight rows up to eight past the fifteen
inline size_t Tc64Plan::smem_syn(int blocks) const {
  const size_t red = static_cast<size_t>(2 * 64 * blocks) * (std::min(lrows, 32) + 1) * sizeof(int);
  return std::max(static_cast<size_t>(ns) * T64_DIG * lrows * 32, red) + static_cast<size_t>(kc_max) * 15 * blocks * T64_SBO + 8 * T64_SBO + 256;
}

// sizes, offsets and tables for members B (the digits are cut on the device from the FP64 tables)
inline void build_tc64(Tc64Plan &p, const HostTables &h, const SphDev &d, double radius, int B, cudaStream_t stream) {
  const int N = h.N, M = h.M, nh = h.nh, ext = h.ntri + M;
  p.nh16 = pad16(nh);
  p.lrows = std::min(p.nh16, 64);
  p.nsl = p.nh16 / p.lrows;
  p.nhk = pad16(nh);
  std::vector<int> ke16(M), kc(M), ra16(2 * M);
  std::vector<long> oS(M), oA(2 * M);
  long ts = 0, ta = 0;
  for (int m = 0; m <= N; m++) {
    const int even = (N + 1 - m) / 2 + 1, odd = (N + 2 - m) / 2;  // n - m = 0..T+1-m
    ke16[m] = pad16(even);
    kc[m] = (ke16[m] + pad16(odd)) / 16;
    p.kc_max = std::max(p.kc_max, kc[m]);
    oS[m] = ts;
    ts += static_cast<long>(p.nsl) * kc[m] * T64_DIG * p.lrows * 16;
    for (int s = 0; s < 2; s++) {
      ra16[2 * m + s] = pad16(s ? odd : even);
      p.ra_max = std::max(p.ra_max, ra16[2 * m + s]);
      oA[2 * m + s] = ta;
      ta += static_cast<long>(p.nhk / 16) * T64_DIG * ra16[2 * m + s] * 16;
    }
  }
  // the coefficients of U, V and of the derivative sums (legendre_eps: cpp/sphere.cpp:11)
  std::vector<double> cf(5 * static_cast<size_t>(ext), 0.0);
  for (int m = 0; m <= N; m++)
    for (int n = m; n <= N + 1; n++) {
      const size_t i = static_cast<size_t>(h.tri[m] + n);
      const double el = n > m ? legendre_eps(n, m) : 0.0, eu = legendre_eps(n + 1, m);
      cf[i] = n > 0 ? radius * m / (n * (n + 1.0)) : 0.0;
      cf[ext + i] = n > 0 ? radius * el / n : 0.0;
      cf[2 * static_cast<size_t>(ext) + i] = radius * eu / (n + 1.0);
      cf[3 * static_cast<size_t>(ext) + i] = n * eu;
      cf[4 * static_cast<size_t>(ext) + i] = (n + 1) * el;
    }
  auto up = [&](auto &dst, const auto &src) {
    dst.alloc(src.size());
    copy_in(dst.p, src.data(), src.size() * sizeof(src[0]), stream);
  };
  up(p.ke16, ke16);
  up(p.kc, kc);
  up(p.ra16, ra16);
  up(p.oS, oS);
  up(p.oA, oA);
  up(p.cf, cf);
  p.tS.alloc(ts);
  p.tA.alloc(ta);
  p.eS.alloc(static_cast<size_t>(M) * p.nh16);
  p.eA.alloc(ext);
  p.err.alloc(1);
  p.err.p[0] = 0;
  // members per synthesis tile: two share an MMA (its 128 rows) where one each would not fit the SMs at once
  p.nbt = B > 1 && static_cast<long>(M) * p.nsl * B > 2 * kSMs ? 2 : 1;
  p.ntiles = (B + p.nbt - 1) / p.nbt;
  // Table chunks in flight: three where several CTAs share an SM and hide one another's waits, else as many as there are
  // and fit, so that all of them have arrived when the predecessor ends
  const auto stages = [](long ctas, size_t a, size_t stage, int chunks) {
    const size_t room = 225 * 1024 / static_cast<size_t>(std::max(1l, std::min(2l, (ctas + kSMs - 1) / kSMs))) - 1024;
    const int fit = room > a ? static_cast<int>((room - a) / stage) : 0;
    return ctas > 2 * kSMs ? 3 : std::max(3, std::min({fit, chunks, T64_STAGES}));
  };
  const size_t a_syn = static_cast<size_t>(p.kc_max) * 30 * T64_SBO + 8 * T64_SBO + 256, a_ana = static_cast<size_t>(2) * (p.nhk / 16) * 30 * T64_SBO;
  p.ns = stages(static_cast<long>(M) * p.nsl * p.ntiles, a_syn, static_cast<size_t>(T64_DIG) * p.lrows * 32, p.kc_max);
  const size_t ana_stage = static_cast<size_t>(T64_DIG) * p.ra_max * 32;
  // an analysis CTA that cannot share its SM (T170's operand) has it alone
  const bool alone = a_ana + 3 * ana_stage > 112 * 1024;
  p.nsa = stages(alone ? 1 : static_cast<long>(M) * B, a_ana, ana_stage, 2 * (p.nhk / 16));
  // 512 threads shorten the digits, the sums and the update of a CTA that shares its SM with at most one other; more CTAs of
  // 256 overlap their phases better (T170 x 4, one CTA per SM: 88.2 us with 256 threads, 82.1 with 512)
  p.wide = alone || static_cast<long>(M) * B <= 2 * kSMs;
  const size_t red_ana = static_cast<size_t>(p.wide ? 4 : 2) * 128 * 33 * sizeof(int) + 16 + static_cast<size_t>(16) * (N + 3) * sizeof(double);
  p.smem_ana = std::max(static_cast<size_t>(p.nsa) * ana_stage + a_ana, red_ana);
  DevBuf<double> P1;
  up(P1, h.P1);
  const Tc64Dev z = tc64_dev(p, ext);
  tc64_build_syn<<<M, 128, 0, stream>>>(d, z, P1.p, p.tS.p, p.eS.p);
  tc64_build_ana<<<dim3(M, 2), 256, 0, stream>>>(d, z, P1.p, p.tA.p, p.eA.p);
  LMW_LAUNCH_CHECK();
  LMW_CUDA(cudaStreamSynchronize(stream));
}

}  // namespace lmw
