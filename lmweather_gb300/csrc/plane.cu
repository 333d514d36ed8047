// Beta-plane C-grid shallow water on the GPU (FP64), the lmweather Plane model (cpp/plane.cpp).
//
// One fused kernel per RK4 stage: a CTA loads a (rows+2) x (TX+2) tile of h, u, v (periodic in x, rows
// clamped at the walls) into shared memory, forms the Bernoulli function B and the absolute vorticity eta
// for the tile plus its one-cell halo, evaluates du, dv, dh, and applies the RK4 stage update in the same
// pass (stage input, accumulator and, at the last stage, the state). Every value is the one the reference's
// order of evaluation gives (plane_stage says where fewer operations give it) and this file is compiled with
// --fmad=false, so that the result is bitwise identical to cpp/plane.cpp:59-158 built without FMA contraction.
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "engine.h"
#include "fixed_div.cuh"

namespace lmw {
namespace {

constexpr int TX = 32;  // tile width: one warp per row of cells

struct PlaneDev {
  int nx, ny, lin;
  double dxx, dyy, dxx2, dyy2, g, depth, f0, beta, visc, drag, ly, hly;  // hly = 0.5 ly (exact)
  double zh[4], zl[4];  // two-term reciprocals of dxx, dyy, dxx2, dyy2 (in that order), for div_fixed
  FixedDiv2 fd[4];      // the same divisors for div_fixed2
  int hasdrag, hasvisc; // drag, viscosity not zero (tested on the integer pipe)
  int fastdiv;          // 2: all four divisors qualify for div_fixed2; 1: they and their reciprocals are normal numbers
};

// what div_fixed2 does not answer: div_fixed when the host found the spacings normal, else IEEE
__device__ __noinline__ double div_general(double x, double y, double zh, double zl, int fastdiv) {
  int fast;
  return fastdiv ? div_fixed(x, y, zh, zl, fast) : x / y;
}
// the stencil's divisions by the grid spacings, K = 0..3: dxx, dyy, dxx2, dyy2
template <int K> __device__ __forceinline__ double div_by(const PlaneDev &p, double x) {
  int ok;
  const double q = div_fixed2(x, p.fd[K], ok);
  if (p.fastdiv == 2 && ok) return q;
  return div_general(x, K == 0 ? p.dxx : K == 1 ? p.dyy : K == 2 ? p.dxx2 : p.dyy2, p.zh[K], p.zl[K], p.fastdiv);
}

// 2^-E <= |x| < 2^E, by integer operations
__device__ __forceinline__ unsigned magnitude(double x) { return static_cast<unsigned>(__double2hiint(x)) & 0x7fffffffu; }
template <int E> __device__ __forceinline__ bool within(double x) {
  return magnitude(x) - (static_cast<unsigned>(1023 - E) << 20) < static_cast<unsigned>(2 * E) << 20;
}
__device__ __forceinline__ bool is_zero(double x) { return (magnitude(x) | static_cast<unsigned>(__double2loint(x))) == 0u; }
__device__ __forceinline__ bool not_finite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }
// What plane_stage leaves to the reference's own operations (see there): q vbar from the sums of two eta and four v, B from g h
// and the sums of squares, and dh at cell (tx, ty) of a tile from its points
__device__ __noinline__ double edge_product(double e2, double s2) { return 0.5 * e2 * (0.25 * s2); }
__device__ __noinline__ double edge_bernoulli(double b, double qx, double qy) { return b + 0.5 * (0.5 * qx + 0.5 * qy); }
__device__ __noinline__ double edge_dh(const PlaneDev &p, const double (*sh)[TX + 2], const double (*su)[TX + 2], const double (*sv)[TX + 2], int tx,
                                       int ty, int j) {
  const double hc = sh[ty + 1][tx + 1];
  const double hw = p.lin ? p.depth : 0.5 * (sh[ty + 1][tx] + hc), he = p.lin ? p.depth : 0.5 * (hc + sh[ty + 1][tx + 2]);
  const double fe = he * su[ty + 1][tx + 2], fw = hw * su[ty + 1][tx + 1];
  double fn = 0, fs = 0;
  if (j + 1 < p.ny) fn = (p.lin ? p.depth : 0.5 * (hc + sh[ty + 2][tx + 1])) * sv[ty + 2][tx + 1];
  if (j > 0) fs = (p.lin ? p.depth : 0.5 * (sh[ty][tx + 1] + hc)) * sv[ty + 1][tx + 1];
  return -(div_general(fe - fw, p.dxx, p.zh[0], p.zl[0], p.fastdiv) + div_general(fn - fs, p.dyy, p.zh[1], p.zl[1], p.fastdiv));
}

// r - drag U. With no drag that is r, but for a U that is not finite (NaN) and the sign of a zero
__device__ __forceinline__ double drag_term(const PlaneDev &p, double r, double U) {
  const bool special = not_finite(U) || (__double2hiint(r) == static_cast<int>(0x80000000u) && __double2loint(r) == 0);
  return p.hasdrag || special ? r - p.drag * U : r;
}

__device__ __forceinline__ int wrapx(int i, int nx) { return ((i % nx) + nx) % nx; }

// stage 0..3 with coefficients c = 0.5 dt, 0.5 dt, dt, dt/6 (cpp/plane.cpp:143-158)
//
// Bound: the FP64 pipe (about 1.7 warp lanes per clock and SM; HBM and L2 are idle beside it), so what counts is the
// number of FP64 instructions. The reference's values are kept bit for bit with fewer of them:
//   - its factors 0.5, 0.25 and 2 are exact, so they are folded into the neighbouring operation (q vbar = 0.125 RN(s1 s2)
//     inside the FMA that subtracts the pressure term; the Bernoulli function's 0.25; the flux's 0.5 in the continuity
//     equation's step, whose accumulator holds k / -0.5; acc + 2 k as an FMA). Where such a product could be subnormal or
//     overflow, and round differently, the reference's own operations are called (edge_*), by tests on the integer pipe:
//     for a sum of squares outside 2^-900 .. 2^900; for a sum of four v outside 2^-330 .. 2^330 or its product with eta's
//     outside 2^-660 .. 2^660, zero apart (then neither factor is subnormal); and for a dh that is not finite or belongs to
//     an h below 2^-600 (the error of a subnormal flux, 2^-1074 / 2^-50 at most, is lost in any other h). The tests cost
//     60 x 30 two per cent (3.53 -> 3.62 us a stage of a run), 200 x 100 and 1024 x 512 nothing;
//   - squares, fluxes and B are formed once per point in shared memory, not once per neighbour;
//   - divisions by the spacings take two operations (div_fixed2) where that is proven, not three;
//   - drag U is left out for drag = 0 (drag_term).
// That is 54 FP64 operations per cell and stage instead of 86 (nonlinear, inviscid).
// A tile is TX x ty_n cells: the CTAs are dealt to the tile columns as evenly as they go, and a column's CTAs cut its
// rows evenly. A tile's 3 TX ty_n updates (u, v, h: one role per warp) are dealt to the NT threads, so a tile of one row
// still has three warps working at once. The base state and the accumulator of a thread's updates are loaded ahead of
// the tile. plane_tiling picks the number of CTAs and the form.
// EARLY: the next stage's CTAs launch while this one's wait for their predecessor (griddepcontrol), which takes the
// launch out of the chain from stage to stage. They are placed where there is room, so every SM has to hold the same
// number of CTAs: with some SMs idle they would pile up there (300 x 200 in 130 tiles: 36 us a stage, against 14 us
// without the early launch). Otherwise the next stage's CTAs launch when the last wave has only its updates left.
// Stage time before and now (us): 60 x 30 12.4 -> 3.8, 200 x 100 14.3 -> 5.3, 1024 x 512 118.9 -> 68.3 (its 54
// operations a cell take 53 at 0.53e12 a second), 4000 x 2000 1678 -> 953.
template <int TYMAX, int NT, bool EARLY>
__global__ void __launch_bounds__(NT, 1024 / NT) plane_stage(const __grid_constant__ PlaneDev p, int stage, double c, const double *coef, const double *hi,
                                                             const double *ui, const double *vi, double *h0, double *u0, double *v0, double *ah,
                                                             double *au, double *av, double *ho, double *uo, double *vo) {
  constexpr int TY = TYMAX;
  __shared__ double sh[TY + 2][TX + 2], su[TY + 2][TX + 2], sv[TY + 2][TX + 2], qu[TY + 2][TX + 2], qv[TY + 2][TX + 2];
  __shared__ double sB[TY + 1][TX + 1], sE[TY + 1][TX + 1], sF[TY][TX + 1], sG[TY + 1][TX], sf[TY + 1];
  constexpr int ITEMS = (3 * TY * TX + NT - 1) / NT;
  const int nx = p.nx, ny = p.ny;
  const int tiles_x = (nx + TX - 1) / TX, ctas = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  const int col = cta * tiles_x / ctas, first = (col * ctas + tiles_x - 1) / tiles_x, rows = ((col + 1) * ctas + tiles_x - 1) / tiles_x - first;
  const int i0 = col * TX, j0 = (cta - first) * ny / rows, ty_n = (cta - first + 1) * ny / rows - j0, ncell = ty_n * TX;
  const int tid = threadIdx.x;
  if (coef != nullptr) c = coef[stage];  // written before the first of a chain of stages
  if (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the updates of this thread: role 0 u, 1 v, 2 h
  double xv[ITEMS], kv[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const int e = tid + k * NT, role = e < ncell ? 0 : e < 2 * ncell ? 1 : e < 3 * ncell ? 2 : 3, w = e - role * ncell;
    const int i = i0 + w % TX, j = j0 + w / TX;
    xv[k] = kv[k] = 0;
    if (role < 3 && i < nx && j < ny) {
      const size_t o = static_cast<size_t>(j) * nx + i;
      xv[k] = role == 0 ? u0[o] : role == 1 ? v0[o] : h0[o];
      if (stage > 0) kv[k] = role == 0 ? au[o] : role == 1 ? av[o] : ah[o];
    }
  }
  // tile load: local (ly, lx) <-> global (j0 - 1 + ly, i0 - 1 + lx), periodic in x; columns past nx are not used
  for (int e = tid; e < (ty_n + 2) * (TX + 2); e += NT) {
    const int ly = e / (TX + 2), lx = e % (TX + 2);
    const int jg = j0 - 1 + ly;
    int ig = i0 - 1 + lx;
    ig = ig < 0 ? ig + nx : ig >= nx ? ig - nx : ig;
    if (ig >= nx) ig = 0;
    double hv = 0, uv = 0, vv = 0;
    if (jg >= 0 && jg < ny) {
      const size_t o = static_cast<size_t>(jg) * nx + ig;
      hv = hi[o];
      uv = ui[o];
    }
    if (jg >= 0 && jg <= ny) vv = vi[static_cast<size_t>(jg) * nx + ig];
    sh[ly][lx] = hv;
    su[ly][lx] = uv;
    sv[ly][lx] = vv;
    if (!p.lin) {
      qu[ly][lx] = uv * uv;
      qv[ly][lx] = vv * vv;
    }
  }
  // the Coriolis parameter of the corner rows
  if (tid >= NT - ty_n - 1) {
    const int ly = tid - (NT - ty_n - 1);
    sf[ly] = p.f0 + p.beta * ((j0 + ly) * p.dyy - p.hly);
  }
  __syncthreads();
  // Bernoulli B at cells (j0-1+ly, i0-1+lx), absolute vorticity at corners (j0+ly, i0+lx), cpp/plane.cpp:70-92, and twice
  // the fluxes of the west faces (j0+ly, i0+lx) and south faces (j0+ly, i0+lx), cpp/plane.cpp:119-128 (the fluxes
  // themselves in the linear model)
  for (int e = tid; e < (ty_n + 1) * (TX + 1); e += NT) {
    const int ly = e / (TX + 1), lx = e % (TX + 1);
    if (i0 + lx > nx || j0 + ly > ny) continue;
    const int jb = j0 - 1 + ly, je = j0 + ly;
    double b = 0;
    if (jb >= 0) {
      b = p.g * sh[ly][lx];
      if (!p.lin) {
        const double qx = qu[ly][lx] + qu[ly][lx + 1], qy = qv[ly][lx] + qv[ly + 1][lx], q = qx + qy;
        if (within<900>(q)) b = __fma_rn(0.25, q, b);
        else b = edge_bernoulli(b, qx, qy);
      }
    }
    sB[ly][lx] = b;
    double zeta = 0;
    if (!p.lin) {
      const double dvdx = div_by<0>(p, sv[ly + 1][lx + 1] - sv[ly + 1][lx]);
      const double uj = je < ny ? su[ly + 1][lx + 1] : su[ly][lx + 1];
      const double ujm = je > 0 ? su[ly][lx + 1] : su[ly + 1][lx + 1];
      zeta = dvdx - div_by<1>(p, uj - ujm);
    }
    sE[ly][lx] = sf[ly] + zeta;
    if (ly < ty_n) {
      const double u = su[ly + 1][lx + 1];
      sF[ly][lx] = p.lin ? p.depth * u : (sh[ly + 1][lx] + sh[ly + 1][lx + 1]) * u;
    }
    if (lx < TX) {
      const double v = sv[ly + 1][lx + 1];
      sG[ly][lx] = je == 0 || je == ny ? 0.0 : p.lin ? p.depth * v : (sh[ly][lx + 1] + sh[ly + 1][lx + 1]) * v;
    }
  }
  __syncthreads();
  if (!EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const double ch = p.lin ? -c : -0.5 * c;  // dh = -0.5 (twice the flux divergence)
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const int e = tid + k * NT, role = e < ncell ? 0 : e < 2 * ncell ? 1 : e < 3 * ncell ? 2 : 3, w = e - role * ncell;
    const int tx = w % TX, ty = w / TX, i = i0 + tx, j = j0 + ty;
    if (role >= 3 || i >= nx || j >= ny) continue;
    double r;
    if (role == 0) {
      // du at the u point (i, j): cpp/plane.cpp:94-105
      const double U = su[ty + 1][tx + 1];
      const double s2 = sv[ty + 1][tx] + sv[ty + 1][tx + 1] + sv[ty + 2][tx] + sv[ty + 2][tx + 1];
      const double e2 = sE[ty][tx] + sE[ty + 1][tx], es = e2 * s2, pr = div_by<0>(p, sB[ty + 1][tx + 1] - sB[ty + 1][tx]);
      if (is_zero(es) || (within<330>(s2) && within<660>(es))) r = __fma_rn(0.125, es, -pr);
      else r = edge_product(e2, s2) - pr;
      r = drag_term(p, r, U);
      if (p.hasvisc) {
        const double uy1 = j + 1 < ny ? su[ty + 2][tx + 1] : U, uy0 = j > 0 ? su[ty][tx + 1] : U;
        r += p.visc * (div_by<2>(p, __fma_rn(-2.0, U, su[ty + 1][tx + 2]) + su[ty + 1][tx]) + div_by<3>(p, __fma_rn(-2.0, U, uy1) + uy0));
      }
    } else if (role == 1) {
      // dv at the v point (i, j), interior rows only: cpp/plane.cpp:106-117
      r = 0;
      if (j >= 1) {
        const double V = sv[ty + 1][tx + 1];
        const double s2 = su[ty][tx + 1] + su[ty][tx + 2] + su[ty + 1][tx + 1] + su[ty + 1][tx + 2];
        const double e2 = sE[ty][tx] + sE[ty][tx + 1], es = e2 * s2, pr = div_by<1>(p, sB[ty + 1][tx + 1] - sB[ty][tx + 1]);
        if (is_zero(es) || (within<330>(s2) && within<660>(es))) r = __fma_rn(-0.125, es, -pr);
        else r = edge_product(-e2, s2) - pr;
        r = drag_term(p, r, V);
        if (p.hasvisc) {
          const double vy1 = j + 1 < ny ? sv[ty + 2][tx + 1] : 0.0, vy0 = j - 1 > 0 ? sv[ty][tx + 1] : 0.0;
          r += p.visc * (div_by<2>(p, __fma_rn(-2.0, V, sv[ty + 1][tx + 2]) + sv[ty + 1][tx]) + div_by<3>(p, __fma_rn(-2.0, V, vy1) + vy0));
        }
      }
    } else {
      r = div_by<0>(p, sF[ty][tx + 1] - sF[ty][tx]) + div_by<1>(p, sG[ty + 1][tx] - sG[ty][tx]);
      if (!p.lin && (not_finite(r) || magnitude(xv[k]) < (423u << 20) || p.fastdiv != 2)) r = -2.0 * edge_dh(p, sh, su, sv, tx, ty, j);
    }
    // RK4 bookkeeping: cpp/plane.cpp:146-156 (acc = k1 + 2 k2 + 2 k3, state += dt/6 (acc + k4)); for h, r = k / -0.5
    // (linear: -k), which its accumulator keeps and its coefficient takes up
    const double cc = role == 2 ? ch : c;
    const size_t o = static_cast<size_t>(j) * nx + i;
    double *out = role == 0 ? uo : role == 1 ? vo : ho, *acc = role == 0 ? au : role == 1 ? av : ah;
    if (stage < 3) {
      out[o] = xv[k] + cc * r;
      acc[o] = stage == 0 ? r : __fma_rn(2.0, r, kv[k]);
      if (role == 1 && j == ny - 1) vo[o + nx] = v0[o + nx];  // the northern wall row ny does not move
    } else {
      (role == 0 ? u0 : role == 1 ? v0 : h0)[o] = xv[k] + cc * (kv[k] + r);
    }
  }
}

// the stage coefficients into device memory (by value: a copy from the host's stack could still be under way when the
// caller has returned)
__global__ void plane_coef(double *c, double half, double full, double sixth) {
  c[0] = c[1] = half;
  c[2] = full;
  c[3] = sixth;
}

// How a grid is cut. FORM 0: at most one one-row tile per SM; 1, 2: one or two CTAs on every SM, tiles of up to sixteen
// rows; 3: more. 0 to 2 launch early. In 3 the rows of a tile are the number up to sixteen that leaves the fullest SM
// the least to do, counting the FP64 instructions per warp of a tile: 2 for each loaded point, 17 for each corner, 33
// for each cell (sixteen rows lose 4 % to the halo, eight 7 %). Measured, us a stage: 200 x 100 in form 1 5.2, 2 7.0,
// 3 8.5; 400 x 200 (too tall for form 1) in 2 13.8, 3 15.1.
constexpr int PLANE_TY = 16;
struct Tiling {
  int form, ctas, ty;  // ty: rows of the tallest tile
};
Tiling plane_tiling(int nx, int ny) {
  const int tx = (nx + TX - 1) / TX;
  if (tx * ny <= kSMs) return {0, tx * ny, 1};
  for (int per_sm = 1; per_sm <= 2; per_sm++) {
    const int least = per_sm * kSMs / tx;  // CTAs of the column with the fewest
    if (least > 0 && (ny + least - 1) / least <= PLANE_TY && (per_sm * kSMs + tx - 1) / tx <= ny)
      return {per_sm, per_sm * kSMs, (ny + least - 1) / least};
  }
  Tiling best{3, 0, 0};
  double bc = 1e300;
  for (int rows = (ny + PLANE_TY - 1) / PLANE_TY; rows <= (ny + 7) / 8; rows++) {
    const int ty = (ny + rows - 1) / rows, load = ((ty + 2) * (TX + 2) + 31) / 32, corner = ((ty + 1) * (TX + 1) + 31) / 32;
    const double cost = static_cast<double>((tx * rows + kSMs - 1) / kSMs) * (2 * load + 17 * corner + 33 * ty);
    if (cost < bc) {
      bc = cost;
      best = {3, tx * rows, ty};
    }
  }
  return best;
}

template <int TY, int NT, bool EARLY, class... A> void plane_launch(const PlaneDev &p, int ctas, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(NT);
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  LMW_CUDA(cudaLaunchKernelEx(&cfg, plane_stage<TY, NT, EARLY>, p, args...));
}
// one RK4 stage with coefficient coef[stage] (device memory; null: c): state (h0, u0, v0), stage input (hi, ui, vi), accumulator, next stage input
void stage_launch(const PlaneDev &p, cudaStream_t s, int stage, double c, const double *coef, const double *hi, const double *ui, const double *vi, double *h0,
                  double *u0, double *v0, double *ah, double *au, double *av, double *ho, double *uo, double *vo) {
  const Tiling t = plane_tiling(p.nx, p.ny);
  auto run = [&](auto ty, auto nt, auto early) {
    plane_launch<decltype(ty)::value, decltype(nt)::value, decltype(early)::value>(p, t.ctas, s, stage, c, coef, hi, ui, vi, h0, u0, v0, ah, au, av, ho, uo,
                                                                                   vo);
  };
  using std::integral_constant;
  const integral_constant<int, PLANE_TY> tall;
  if (t.form == 0) run(integral_constant<int, 1>(), integral_constant<int, 128>(), std::true_type());
  // one CTA per SM: sixteen warps (97 x 160: 5.2 us a stage against 7.2 with eight; 100 x 64: 4.0 against 4.2)
  else if (t.form == 1) run(tall, integral_constant<int, 512>(), std::true_type());
  else if (t.form == 2) run(tall, integral_constant<int, 256>(), std::true_type());
  else run(tall, integral_constant<int, 256>(), std::false_type());
}

// ---------------------------------------------------------------- reductions (guards and diagnostics)
// per block: sum h, sum u, sum v, energy sum, pv^2 sum; max speed, max h
constexpr int RED_THREADS = 256;
constexpr int RED_SUMS = 5, RED_MAXS = 2;

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

__global__ void __launch_bounds__(RED_THREADS) plane_reduce(PlaneDev p, const double *__restrict__ h, const double *__restrict__ u,
                                                            const double *__restrict__ v, double *part) {
  const int nx = p.nx, ny = p.ny;
  const size_t ncell = static_cast<size_t>(nx) * ny, nv = static_cast<size_t>(nx) * (ny + 1);
  double s[RED_SUMS] = {0, 0, 0, 0, 0}, mx[RED_MAXS] = {0, -INFINITY};
  for (size_t e = blockIdx.x * (size_t)RED_THREADS + threadIdx.x; e < nv; e += (size_t)gridDim.x * RED_THREADS) {
    s[2] += v[e];
    if (e >= ncell) continue;
    int j = static_cast<int>(e / nx), i = static_cast<int>(e % nx);
    double hh = h[e];
    s[0] += hh;
    s[1] += u[e];
    double uc = 0.5 * (u[e] + u[static_cast<size_t>(j) * nx + (i + 1) % nx]);
    double vc = 0.5 * (v[e] + v[e + nx]);
    s[3] += 0.5 * hh * (uc * uc + vc * vc) + 0.5 * p.g * hh * hh;
    mx[0] = fmax(mx[0], hypot(uc, vc));
    mx[1] = fmax(mx[1], hh);
    if (j >= 1) {  // PV anomaly at interior corners, cpp/plane.cpp:228-243
      int im = (i + nx - 1) % nx;
      double hav = 0.25 * (h[static_cast<size_t>(j - 1) * nx + im] + h[static_cast<size_t>(j - 1) * nx + i] +
                           h[static_cast<size_t>(j) * nx + im] + hh);
      double dvdx = (v[e] - v[static_cast<size_t>(j) * nx + im]) / p.dxx;
      double z = dvdx - (u[e] - u[e - nx]) / p.dyy;
      double q = z - p.f0 * (hav - p.depth) / p.depth;
      s[4] += q * q;
    }
  }
  __shared__ double red[RED_THREADS / 32][RED_SUMS + RED_MAXS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int k = 0; k < RED_SUMS; k++) s[k] = warp_sum(s[k]);
  for (int k = 0; k < RED_MAXS; k++) mx[k] = warp_max(mx[k]);
  if (lane == 0) {
    for (int k = 0; k < RED_SUMS; k++) red[wid][k] = s[k];
    for (int k = 0; k < RED_MAXS; k++) red[wid][RED_SUMS + k] = mx[k];
  }
  __syncthreads();
  if (threadIdx.x < RED_SUMS + RED_MAXS) {
    int k = threadIdx.x;
    double a = red[0][k];
    for (int w = 1; w < RED_THREADS / 32; w++) a = k < RED_SUMS ? a + red[w][k] : fmax(a, red[w][k]);
    part[static_cast<size_t>(blockIdx.x) * (RED_SUMS + RED_MAXS) + k] = a;
  }
}

__global__ void plane_reduce_final(const double *part, int nblk, Reduce *out) {
  int k = threadIdx.x;
  if (k >= RED_SUMS + RED_MAXS) return;
  double a = part[k];
  for (int b = 1; b < nblk; b++) {
    double x = part[static_cast<size_t>(b) * (RED_SUMS + RED_MAXS) + k];
    a = k < RED_SUMS ? a + x : fmax(a, x);
  }
  if (k < RED_SUMS) out->sum[k] = a;
  else out->max[k - RED_SUMS] = a;
}

// ---------------------------------------------------------------- point and harmonic diagnostics
// One thread: kind 0..2 -> bilinear value of h, u or v at (x, y) (cpp/plane.cpp:245-264: each field on its own
// points, periodic in x, rows clamped); kind 3 -> relative vorticity at corner (ci, cj) (cpp/plane.cpp:220-226).
// Compiled without FMA contraction, so the value is the reference's bit for bit.
__global__ void plane_point(PlaneDev p, const double *__restrict__ h, const double *__restrict__ u, const double *__restrict__ v, int kind,
                            double x, double y, int ci, int cj, double *out) {
  const int nx = p.nx, ny = p.ny;
  if (kind == 3) {
    const int im = (ci + nx - 1) % nx;
    const double dvdx = (v[static_cast<size_t>(cj) * nx + ci % nx] - v[static_cast<size_t>(cj) * nx + im]) / p.dxx;
    const double uj = cj < ny ? u[static_cast<size_t>(cj) * nx + ci % nx] : u[static_cast<size_t>(ny - 1) * nx + ci % nx];
    const double ujm = cj > 0 ? u[static_cast<size_t>(cj - 1) * nx + ci % nx] : u[ci % nx];
    out[0] = dvdx - (uj - ujm) / p.dyy;
    return;
  }
  const double xs = kind == 1 ? 0.0 : 0.5, ys = kind == 2 ? 0.0 : 0.5;
  const double fx = x / p.dxx - xs, fy = y / p.dyy - ys;
  const int rows = kind == 2 ? ny + 1 : ny;
  const double fl = floor(fx);
  const int i0 = static_cast<int>(fl), j0 = static_cast<int>(floor(fy));
  const double ax = fx - fl, ay = fy - floor(fy);
  const double *f = kind == 0 ? h : kind == 1 ? u : v;
  auto get = [&](int i, int j) {
    i = wrapx(i, nx);
    j = max(0, min(rows - 1, j));
    return f[static_cast<size_t>(j) * nx + i];
  };
  out[0] = (1 - ax) * ((1 - ay) * get(i0, j0) + ay * get(i0, j0 + 1)) + ax * ((1 - ay) * get(i0 + 1, j0) + ay * get(i0 + 1, j0 + 1));
}

constexpr int HARM_THREADS = 256;
constexpr double kPiPlane = 3.14159265358979323846;

// one CTA per row: c_m = (1/nx) sum_i f_i exp(-2 pi i m (i + shift) / nx) of rows j0.. of f (cpp/plane.cpp:266-270);
// out[r] = (re, im)
__global__ void __launch_bounds__(HARM_THREADS) plane_row_harmonics(const double *__restrict__ f, int nx, int j0, int m, double shift,
                                                                    double2 *out) {
  __shared__ double red[2][HARM_THREADS / 32];
  const double *row = f + static_cast<size_t>(j0 + blockIdx.x) * nx;
  double cr = 0, ci = 0;
  for (int i = threadIdx.x; i < nx; i += HARM_THREADS) {
    const double th = -2 * kPiPlane * m * (i + shift) / nx;
    double sn, cs;
    sincos(th, &sn, &cs);
    cr += row[i] * cs;
    ci += row[i] * sn;
  }
  cr = warp_sum(cr);
  ci = warp_sum(ci);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][wid] = cr;
    red[1][wid] = ci;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0;
    for (int w = 0; w < HARM_THREADS / 32; w++) {
      a += red[0][w];
      b += red[1][w];
    }
    out[blockIdx.x] = make_double2(a / static_cast<double>(nx), b / static_cast<double>(nx));
  }
}

// sum over rows of |c_m|^2 divided by ny (cpp/plane.cpp:291-299), one thread in row order
__global__ void plane_harmonic_energy_sum(const double2 *__restrict__ c, int rows, int ny, double *out) {
  double s = 0;
  for (int r = 0; r < rows; r++) s += c[r].x * c[r].x + c[r].y * c[r].y;
  out[0] = s / ny;
}

// the divisors of the stencil: dx, dy and their squares
struct Divisors {
  FixedDiv2 fd[4];
  bool proven = true;
};
Divisors make_divisors(const PlaneConfig &c) {
  const double dx = c.lx / c.nx, dy = c.ly / c.ny, dv[4] = {dx, dy, dx * dx, dy * dy};
  Divisors d;
  for (int k = 0; k < 4; k++)
    if (!fixed_div2_setup(dv[k], d.fd[k])) d.proven = false;
  return d;
}

PlaneDev make_dev(const PlaneConfig &c, const Divisors &div) {
  PlaneDev d;
  d.nx = c.nx;
  d.ny = c.ny;
  d.lin = c.linear ? 1 : 0;
  d.dxx = c.lx / c.nx;
  d.dyy = c.ly / c.ny;
  d.dxx2 = d.dxx * d.dxx;
  d.dyy2 = d.dyy * d.dyy;
  d.g = c.gravity;
  d.depth = c.depth;
  d.f0 = c.f0;
  d.beta = c.beta;
  d.visc = c.viscosity;
  d.drag = c.drag;
  d.ly = c.ly;
  d.hly = 0.5 * c.ly;
  d.hasdrag = c.drag != 0 ? 1 : 0;
  d.hasvisc = c.viscosity != 0 ? 1 : 0;
  const double dv[4] = {d.dxx, d.dyy, d.dxx2, d.dyy2};
  d.fastdiv = 1;
  for (int k = 0; k < 4; k++) {
    if (!fixed_div_reciprocal(dv[k], d.zh[k], d.zl[k])) d.fastdiv = 0;
    d.fd[k] = div.fd[k];
  }
  if (d.fastdiv && div.proven) d.fastdiv = 2;
  return d;
}

// splitmix64 and the Irwin-Hall normal of cpp/plane.cpp:12-17,37-41 (host, for the seeded initialisers)
uint64_t splitmix(uint64_t &x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
double irwin_hall(uint64_t &st) {
  double s = 0;
  for (int i = 0; i < 12; i++) s += static_cast<double>(splitmix(st) >> 11) * (1.0 / 9007199254740992.0);
  return s - 6.0;
}

// Scratch of lmw_plane_step_noalloc: the two RK4 stage inputs and the accumulator (three fields each), in
// device memory reserved when the library is loaded, so that the entry point never allocates. Each field slot
// holds kNoAllocFieldCap doubles: up to kNoAllocMaxCells cells for h and u, plus one row (nx <= 4000) for v.
constexpr size_t kNoAllocMaxCells = 262144;
constexpr size_t kNoAllocFieldCap = kNoAllocMaxCells + 4096;
static __device__ __align__(256) double g_noalloc_scratch[9 * kNoAllocFieldCap];

// div_fixed and the stencil's division against the IEEE division on every pair (x[i], y[k]): counts[0] = results that differ in any bit,
// counts[1] = pairs div_fixed's fast path answered (the rest took the IEEE division)
__global__ void division_selftest(const unsigned long long *__restrict__ xb, int nx, const double *__restrict__ y,
                                  const double *__restrict__ zh, const double *__restrict__ zl, const FixedDiv2 *__restrict__ fd, int ny,
                                  unsigned long long *counts) {
  const long long total = static_cast<long long>(nx) * ny;
  unsigned long long bad = 0, fastn = 0;
  // the stencil's division: two operations where they are proven, else div_general (zh = 0: not proven for this divisor)
  auto differs = [&](double x, int k) {
    int ok = 0;
    double q = fd[k].zh != 0 ? div_fixed2(x, fd[k], ok) : 0.0;
    if (!ok) q = div_general(x, y[k], zh[k], zl[k], 1);
    return __double_as_longlong(q) != __double_as_longlong(x / y[k]);
  };
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const double x = __longlong_as_double(static_cast<long long>(xb[e % nx]));
    const int k = static_cast<int>(e / nx);
    int fast = 0;
    const double a = div_fixed(x, y[k], zh[k], zl[k], fast);
    const double b = x / y[k];
    bad += __double_as_longlong(a) != __double_as_longlong(b) || differs(x, k) ? 1 : 0;
    fastn += fast;
  }
  // each divisor's own exceptional dividend
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ny; k += gridDim.x * blockDim.x)
    for (int e = 1023 - 3; fd[k].zh != 0 && fd[k].bad_hi < 1u << 20 && e < 1023 + 4; e++) {
      const double x = __hiloint2double(static_cast<int>(static_cast<unsigned>(e) << 20 | fd[k].bad_hi), static_cast<int>(fd[k].bad_lo));
      bad += differs(x, k) || differs(-x, k) ? 1 : 0;
    }
  if (bad) atomicAdd(&counts[0], bad);
  if (fastn) atomicAdd(&counts[1], fastn);
}

}  // namespace

struct PlaneDivisors : Divisors {};

void division_selftest_run(const uint64_t *x, int nx, const double *y, int ny, long long *counts) {
  if (nx < 0 || ny < 0 || nx > (1 << 26) || ny > 4096) throw InvalidArgument("counts out of range");
  std::vector<double> zh(std::max(ny, 1)), zl(std::max(ny, 1));
  for (int k = 0; k < ny; k++)
    if (!fixed_div_reciprocal(y[k], zh[k], zl[k]))
      throw InvalidArgument("divisor " + std::to_string(k) + " or its reciprocal is not a normal number");
  std::vector<FixedDiv2> fd(std::max(ny, 1));
  for (int k = 0; k < ny; k++)
    if (!fixed_div2_setup(y[k], fd[k])) fd[k].zh = 0;
  DevBuf<unsigned long long> xd, cd;
  DevBuf<double> yd, hd, ld;
  DevBuf<FixedDiv2> fdd;
  fdd.alloc(fd.size());
  xd.alloc(std::max(nx, 1));
  yd.alloc(std::max(ny, 1));
  hd.alloc(std::max(ny, 1));
  ld.alloc(std::max(ny, 1));
  cd.alloc(2);
  if (nx) LMW_CUDA(cudaMemcpy(xd.p, x, nx * sizeof(unsigned long long), cudaMemcpyHostToDevice));
  if (ny) {
    LMW_CUDA(cudaMemcpy(yd.p, y, ny * sizeof(double), cudaMemcpyHostToDevice));
    LMW_CUDA(cudaMemcpy(hd.p, zh.data(), ny * sizeof(double), cudaMemcpyHostToDevice));
    LMW_CUDA(cudaMemcpy(ld.p, zl.data(), ny * sizeof(double), cudaMemcpyHostToDevice));
    LMW_CUDA(cudaMemcpy(fdd.p, fd.data(), ny * sizeof(FixedDiv2), cudaMemcpyHostToDevice));
  }
  LMW_CUDA(cudaMemset(cd.p, 0, 2 * sizeof(unsigned long long)));
  if (nx > 0 && ny > 0) {
    division_selftest<<<1024, 256>>>(xd.p, nx, yd.p, hd.p, ld.p, fdd.p, ny, cd.p);
    LMW_LAUNCH_CHECK();
    g_launches += 1;
  }
  unsigned long long c[2];
  LMW_CUDA(cudaMemcpy(c, cd.p, sizeof(c), cudaMemcpyDeviceToHost));
  for (int k = 0; k < 2; k++) counts[k] = static_cast<long long>(c[k]);
}

// Device address of g_noalloc_scratch in the calling thread's current CUDA context. In host code the symbol's
// name is only a host-side stand-in, never a device address. A module's globals live in one context: after
// cudaDeviceReset, or in a second context made on the same device with the driver API, the array is loaded
// again at another address. So the address is cached per context (keyed by the driver's unique context id,
// which is never reused within a process) and looked up, with that context current, on the first call made
// in it.
using CtxGetCurrentFn = int (*)(void **);
using CtxGetIdFn = int (*)(void *, unsigned long long *);
static unsigned long long current_context_id() {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<CtxGetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(f);
  });
  if (!get_current || !get_id) throw DeviceError("lmw_plane_step_noalloc: the driver offers no context id (cuCtxGetId)");
  void *ctx = nullptr;
  if (get_current(&ctx) != 0) throw DeviceError("lmw_plane_step_noalloc: cuCtxGetCurrent failed");
  if (ctx == nullptr) {
    // no context bound to this thread yet: a runtime call on the module binds the device's primary context
    void *p = nullptr;
    LMW_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    if (get_current(&ctx) != 0 || ctx == nullptr) throw DeviceError("lmw_plane_step_noalloc: no current CUDA context");
  }
  unsigned long long id = 0;
  if (get_id(ctx, &id) != 0) throw DeviceError("lmw_plane_step_noalloc: cuCtxGetId failed");
  return id;
}

static double *noalloc_scratch() {
  static std::mutex mu;
  static std::vector<std::pair<unsigned long long, double *>> cache;  // (context id, array address)
  const unsigned long long id = current_context_id();
  std::lock_guard<std::mutex> lock(mu);
  for (const auto &e : cache)
    if (e.first == id) return e.second;
  void *p = nullptr;
  LMW_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
  cache.emplace_back(id, static_cast<double *>(p));
  return static_cast<double *>(p);
}

void plane_step_noalloc(const PlaneConfig &c, double *h, double *u, double *v, double dt, int steps, cudaStream_t stream) {
  if (c.nx < 4 || c.ny < 4 || c.nx > 4000 || c.ny > 4000 || static_cast<int64_t>(c.nx) * c.ny > 8000000)
    throw InvalidArgument("grid must be at least 4 x 4 and at most 8 million cells");
  if (!(c.lx > 0 && c.ly > 0)) throw InvalidArgument("domain sizes must be positive");
  const size_t cells = static_cast<size_t>(c.nx) * c.ny;
  if (cells > kNoAllocMaxCells)
    throw InvalidArgument("lmw_plane_step_noalloc: the grid has " + std::to_string(cells) + " cells; this entry point's fixed scratch holds at most " +
                          std::to_string(kNoAllocMaxCells) + " cells (use lmw_plane_create for larger grids)");
  if (!h || !u || !v) throw InvalidArgument("lmw_plane_step_noalloc: field pointer is null");
  if (steps < 0) throw InvalidArgument("lmw_plane_step_noalloc: steps must not be negative");
  if (!std::isfinite(dt)) throw InvalidArgument("lmw_plane_step_noalloc: dt must be finite");
  double *sc = noalloc_scratch();
  // rows 0 and ny of v are the walls; the model keeps them at zero (lmw_plane_set_v does the same), and a
  // nonzero value there would never be cleared (dv = 0 on the walls) and would enter the fluxes and vorticity
  LMW_CUDA(cudaMemsetAsync(v, 0, static_cast<size_t>(c.nx) * sizeof(double), stream));
  LMW_CUDA(cudaMemsetAsync(v + static_cast<size_t>(c.ny) * c.nx, 0, static_cast<size_t>(c.nx) * sizeof(double), stream));
  double *ha = sc, *ua = sc + kNoAllocFieldCap, *va = sc + 2 * kNoAllocFieldCap;
  double *hb = sc + 3 * kNoAllocFieldCap, *ub = sc + 4 * kNoAllocFieldCap, *vb = sc + 5 * kNoAllocFieldCap;
  double *ah = sc + 6 * kNoAllocFieldCap, *au = sc + 7 * kNoAllocFieldCap, *av = sc + 8 * kNoAllocFieldCap;
  // every stage-0 launch writes all of a and the accumulator before any later stage reads them: nothing in the
  // scratch has to start at zero
  PlaneDev d = make_dev(c, make_divisors(c));
  const double half = 0.5 * dt, c6 = dt / 6;
  for (int s = 0; s < steps; s++) {
    stage_launch(d, stream, 0, half, nullptr, h, u, v, h, u, v, ah, au, av, ha, ua, va);
    stage_launch(d, stream, 1, half, nullptr, ha, ua, va, h, u, v, ah, au, av, hb, ub, vb);
    stage_launch(d, stream, 2, dt, nullptr, hb, ub, vb, h, u, v, ah, au, av, ha, ua, va);
    stage_launch(d, stream, 3, c6, nullptr, ha, ua, va, h, u, v, ah, au, av, nullptr, nullptr, nullptr);
    LMW_LAUNCH_CHECK();
    g_launches += 4;
  }
}

PlaneEngine::PlaneEngine(const PlaneConfig &c) : p(c) {
  // cpp/plane.cpp:20-25
  if (c.nx < 4 || c.ny < 4 || c.nx > 4000 || c.ny > 4000 || static_cast<int64_t>(c.nx) * c.ny > 8000000)
    throw InvalidArgument("grid must be at least 4 x 4 and at most 8 million cells");
  if (!(c.lx > 0 && c.ly > 0)) throw InvalidArgument("domain sizes must be positive");
  div = std::make_shared<const PlaneDivisors>(PlaneDivisors{make_divisors(c)});
  LMW_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  coef.alloc(4);
  for (DevBuf<double> *b : {&h0, &u0, &ha, &ua, &hb, &ub, &ah, &au}) b->alloc(ncell());
  for (DevBuf<double> *b : {&v0, &va, &vb, &av}) b->alloc(nvpt());
  nblk_red = 2 * kSMs;
  part.alloc(static_cast<size_t>(nblk_red) * (RED_SUMS + RED_MAXS));
  dred.alloc(1);
  hred.alloc(1);
  stage.alloc(nvpt());
  diag.alloc(2 + 4 * static_cast<size_t>(c.ny));  // one scalar, then a complex per row of u and v
  reset();
}

PlaneEngine::~PlaneEngine() {
  if (graph) cudaGraphExecDestroy(graph);
  if (stream) {
    cudaStreamSynchronize(stream);
    cudaStreamDestroy(stream);
  }
}

void PlaneEngine::upload(double *dst, const double *src, size_t n) {
  for (size_t off = 0; off < n; off += stage.n) {
    size_t c = std::min(stage.n, n - off);
    LMW_CUDA(cudaStreamSynchronize(stream));
    std::memcpy(stage.p, src + off, c * sizeof(double));
    LMW_CUDA(cudaMemcpyAsync(dst + off, stage.p, c * sizeof(double), cudaMemcpyHostToDevice, stream));
  }
  LMW_CUDA(cudaStreamSynchronize(stream));
}

// cpp/plane.cpp:27-32
void PlaneEngine::reset() {
  std::vector<double> hh(ncell(), p.depth);
  upload(h0.p, hh.data(), ncell());
  u0.zero(stream);
  v0.zero(stream);
  LMW_CUDA(cudaStreamSynchronize(stream));
  t = 0;
}

// cpp/plane.cpp:312-318
void PlaneEngine::set_h(const double *g, size_t n) {
  if (n != ncell()) throw InvalidArgument("grid size mismatch");
  upload(h0.p, g, n);
}
void PlaneEngine::set_u(const double *g, size_t n) {
  if (n != ncell()) throw InvalidArgument("grid size mismatch");
  upload(u0.p, g, n);
}
void PlaneEngine::set_v(const double *g, size_t n) {
  if (n != nvpt()) throw InvalidArgument("grid size mismatch");
  std::vector<double> vv(g, g + n);
  for (int i = 0; i < p.nx; i++) {
    vv[i] = 0;
    vv[static_cast<size_t>(p.ny) * p.nx + i] = 0;
  }
  upload(v0.p, vv.data(), n);
}

void PlaneEngine::get(double *h, double *u, double *v) {
  if (h) prefault(h, ncell() * sizeof(double));
  if (u) prefault(u, ncell() * sizeof(double));
  if (v) prefault(v, nvpt() * sizeof(double));
  LMW_CUDA(cudaStreamSynchronize(stream));
  if (h) LMW_CUDA(cudaMemcpy(h, h0.p, ncell() * sizeof(double), cudaMemcpyDeviceToHost));
  if (u) LMW_CUDA(cudaMemcpy(u, u0.p, ncell() * sizeof(double), cudaMemcpyDeviceToHost));
  if (v) LMW_CUDA(cudaMemcpy(v, v0.p, nvpt() * sizeof(double), cudaMemcpyDeviceToHost));
}

// cpp/plane.cpp:34-57: seeded smooth noise. An initialiser, run once on the host in the reference's
// operation order (bitwise identical), then added to the device height.
void PlaneEngine::perturb(double amplitude, uint64_t seed) {
  const int nx = p.nx, ny = p.ny;
  const size_t N = ncell();
  uint64_t st = seed * 0x9E3779B97F4A7C15ULL + 777;
  std::vector<double> n(N), tt(N), h(N);
  for (auto &x : n) x = irwin_hall(st);
  for (int pass = 0; pass < 3; pass++) {
    for (int j = 0; j < ny; j++)
      for (int i = 0; i < nx; i++)
        tt[static_cast<size_t>(j) * nx + i] = 0.25 * n[static_cast<size_t>(j) * nx + (i + nx - 1) % nx] + 0.5 * n[static_cast<size_t>(j) * nx + i] +
                                              0.25 * n[static_cast<size_t>(j) * nx + (i + 1) % nx];
    for (int j = 0; j < ny; j++)
      for (int i = 0; i < nx; i++) {
        int jm = std::max(j - 1, 0), jp = std::min(j + 1, ny - 1);
        n[static_cast<size_t>(j) * nx + i] = 0.25 * tt[static_cast<size_t>(jm) * nx + i] + 0.5 * tt[static_cast<size_t>(j) * nx + i] +
                                             0.25 * tt[static_cast<size_t>(jp) * nx + i];
      }
  }
  double mean = 0, ms = 0;
  for (double x : n) mean += x;
  mean /= n.size();
  for (double &x : n) {
    x -= mean;
    ms += x * x;
  }
  double rms = std::sqrt(ms / n.size());
  double scale = rms > 0 ? amplitude / rms : 0;
  get(h.data(), nullptr, nullptr);
  for (size_t i = 0; i < N; i++) h[i] += n[i] * scale;
  upload(h0.p, h.data(), N);
}

// Zonal jet in geostrophic balance plus white height noise (this project's benchmark initialiser; the same
// definition as the oracle's or_plane_jet_grids).
void PlaneEngine::jet(double u0v, double width, double noise_rms, uint64_t seed) {
  const int nx = p.nx, ny = p.ny;
  const double dyy = dy();
  auto cor = [&](double y) { return p.f0 + p.beta * (y - 0.5 * p.ly); };
  std::vector<double> prof(ny), hy(ny);
  for (int j = 0; j < ny; j++) {
    double y = (j + 0.5) * dyy;
    double c = std::cosh((y - 0.5 * p.ly) / width);
    prof[j] = u0v / (c * c);
  }
  hy[0] = 0;
  for (int j = 1; j < ny; j++) {
    double fa = cor((j - 0.5) * dyy) * prof[j - 1], fb = cor((j + 0.5) * dyy) * prof[j];
    hy[j] = hy[j - 1] - dyy / p.gravity * 0.5 * (fa + fb);
  }
  double mean = 0;
  for (int j = 0; j < ny; j++) mean += hy[j];
  mean /= ny;
  const size_t N = ncell();
  std::vector<double> noise(N), h(N), u(N);
  uint64_t st = seed * 0x9E3779B97F4A7C15ULL + 777;
  for (auto &x : noise) x = irwin_hall(st);
  double nm = 0, ms = 0;
  for (double x : noise) nm += x;
  nm /= N;
  for (double &x : noise) {
    x -= nm;
    ms += x * x;
  }
  double rms = std::sqrt(ms / N);
  double sc = rms > 0 ? noise_rms / rms : 0;
  for (int j = 0; j < ny; j++)
    for (int i = 0; i < nx; i++) {
      size_t k = static_cast<size_t>(j) * nx + i;
      h[k] = p.depth + (hy[j] - mean) + noise[k] * sc;
      u[k] = prof[j];
    }
  upload(h0.p, h.data(), N);
  upload(u0.p, u.data(), N);
  v0.zero(stream);
  LMW_CUDA(cudaStreamSynchronize(stream));
  t = 0;
}

// One RK4 step. cdev: the stage coefficients in device memory (the captured graph, which serves every step size), or
// null: those of dt by value
void PlaneEngine::enqueue_stages(double dt, const double *cdev) {
  const PlaneDev d = make_dev(p, *div);
  const double half = 0.5 * dt, c6 = dt / 6;
  // stage inputs: x0 -> a -> b -> a
  stage_launch(d, stream, 0, half, cdev, h0.p, u0.p, v0.p, h0.p, u0.p, v0.p, ah.p, au.p, av.p, ha.p, ua.p, va.p);
  stage_launch(d, stream, 1, half, cdev, ha.p, ua.p, va.p, h0.p, u0.p, v0.p, ah.p, au.p, av.p, hb.p, ub.p, vb.p);
  stage_launch(d, stream, 2, dt, cdev, hb.p, ub.p, vb.p, h0.p, u0.p, v0.p, ah.p, au.p, av.p, ha.p, ua.p, va.p);
  stage_launch(d, stream, 3, c6, cdev, ha.p, ua.p, va.p, h0.p, u0.p, v0.p, ah.p, au.p, av.p, nullptr, nullptr, nullptr);
  g_launches += 4;
}

void PlaneEngine::enqueue_step(double dt) { enqueue_stages(dt, nullptr); }

void PlaneEngine::set_params(double gravity, double depth, double f0, double beta, double viscosity, double drag, bool linear) {
  p.gravity = gravity;
  p.depth = depth;
  p.f0 = f0;
  p.beta = beta;
  p.viscosity = viscosity;
  p.drag = drag;
  p.linear = linear;
  if (graph) cudaGraphExecDestroy(graph);  // it holds the parameters it was captured with
  graph = nullptr;
}

// `steps` RK4 steps: graphs of GRAPH_STEPS steps (captured once per set of parameters), the rest launched singly
void PlaneEngine::launch_chunk(double dt, int steps) {
  if (steps >= GRAPH_STEPS && coef_dt != dt) {
    plane_coef<<<1, 1, 0, stream>>>(coef.p, 0.5 * dt, dt, dt / 6);
    LMW_LAUNCH_CHECK();
    g_launches += 1;
    coef_dt = dt;
  }
  for (; steps >= GRAPH_STEPS; steps -= GRAPH_STEPS) {
    if (!graph) {
      cudaGraph_t g;
      const uint64_t before = g_launches;
      LMW_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
      for (int s = 0; s < GRAPH_STEPS; s++) enqueue_stages(0.0, coef.p);
      LMW_CUDA(cudaStreamEndCapture(stream, &g));
      g_launches = before;
      LMW_CUDA(cudaGraphInstantiate(&graph, g, 0));
      cudaGraphDestroy(g);
    }
    LMW_CUDA(cudaGraphLaunch(graph, stream));
    g_launches += 4ull * GRAPH_STEPS;
  }
  for (int s = 0; s < steps; s++) enqueue_stages(dt, nullptr);
}

double PlaneEngine::kernel_time(double dt, int reps) {
  PlaneDev d = make_dev(p, *div);
  cudaEvent_t e0, e1;
  LMW_CUDA(cudaEventCreate(&e0));
  LMW_CUDA(cudaEventCreate(&e1));
  // stage 1 reads the base state and stage input a, writes stage input b and the accumulator: x0 is untouched
  stage_launch(d, stream, 1, 0.5 * dt, nullptr, ha.p, ua.p, va.p, h0.p, u0.p, v0.p, ah.p, au.p, av.p, hb.p, ub.p, vb.p);
  LMW_CUDA(cudaEventRecord(e0, stream));
  for (int r = 0; r < reps; r++)
    stage_launch(d, stream, 1, 0.5 * dt, nullptr, ha.p, ua.p, va.p, h0.p, u0.p, v0.p, ah.p, au.p, av.p, hb.p, ub.p, vb.p);
  LMW_CUDA(cudaEventRecord(e1, stream));
  LMW_LAUNCH_CHECK();
  LMW_CUDA(cudaEventSynchronize(e1));
  float ms = 0;
  LMW_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  g_launches += reps + 1;
  return ms / reps;
}

void PlaneEngine::step(double dt) {
  enqueue_step(dt);
  t += dt;
  LMW_CUDA(cudaStreamSynchronize(stream));
}

void PlaneEngine::reduce(Reduce &r) {
  PlaneDev d = make_dev(p, *div);
  plane_reduce<<<nblk_red, RED_THREADS, 0, stream>>>(d, h0.p, u0.p, v0.p, part.p);
  plane_reduce_final<<<1, 32, 0, stream>>>(part.p, nblk_red, dred.p);
  LMW_LAUNCH_CHECK();
  g_launches += 2;
  LMW_CUDA(cudaMemcpyAsync(hred.p, dred.p, sizeof(Reduce), cudaMemcpyDeviceToHost, stream));
  LMW_CUDA(cudaStreamSynchronize(stream));
  r = *hred.p;
}

// cpp/plane.cpp:131-141
double PlaneEngine::stable_dt(double safety) {
  Reduce r;
  if (!p.linear) reduce(r);
  return stable_from(r, safety);
}

// the same from a reduction of the present state (the linear model needs none)
double PlaneEngine::stable_from(const Reduce &r, double safety) const {
  double hmax = p.linear ? p.depth : 0, umax = 0;
  if (!p.linear) {
    umax = r.max[0];
    hmax = std::max(hmax, r.max[1]);
  }
  if (!(hmax > 0)) throw RuntimeError("the depth must be positive to step the model");
  double c = std::sqrt(p.gravity * hmax) + umax;
  double inv = c * std::sqrt(1.0 / (dx() * dx()) + 1.0 / (dy() * dy()));
  double visc = p.viscosity * (4.0 / (dx() * dx()) + 4.0 / (dy() * dy()));
  return safety * 2.0 / (inv + visc + std::fabs(p.f0) + std::fabs(p.beta) * p.ly);
}

// cpp/plane.cpp:160-189
void PlaneEngine::run(double seconds, double dt) {
  if (!(seconds >= 0)) throw InvalidArgument("run: seconds must not be negative");
  if (seconds == 0) return;
  // one reduction gives the automatic step and the limit
  Reduce r;
  if (!p.linear) reduce(r);
  if (!(dt > 0)) dt = stable_from(r, 0.5);
  const double limit = stable_from(r, std::sqrt(0.5));
  if (!(dt <= limit))
    throw InvalidArgument("run: dt = " + fmt_f(dt) + " s exceeds the RK4 stability limit of about " + fmt_f(limit) +
                          " s for the present state: use a smaller dt");
  int64_t n = static_cast<int64_t>(std::ceil(seconds / dt - 1e-9));
  if (n < 1) n = 1;
  if (n > 200000000) throw InvalidArgument("run: too many steps; use a larger dt");
  double hstep = seconds / static_cast<double>(n);
  int64_t i = 0;
  while (i < n) {
    // steps up to and including the next guard point ((i & 63) == 63 or the last step)
    int64_t next = std::min<int64_t>(n - 1, i | 63);
    int chunk = static_cast<int>(next - i + 1);
    launch_chunk(hstep, chunk);
    for (int s = 0; s < chunk; s++) t += hstep;
    i = next + 1;
    reduce(r);
    double s = r.sum[0] + r.sum[1] + r.sum[2];
    if (!std::isfinite(s)) throw RuntimeError("the integration blew up (not finite): use a smaller dt");
    const double now = stable_from(r, std::sqrt(0.5));
    if (!(hstep <= now))
      throw RuntimeError("run: dt = " + fmt_f(hstep) + " s exceeds the RK4 stability limit of about " + fmt_f(now) + " s reached at t = " +
                         fmt_f(t) + " s (the flow accelerated): use a smaller dt");
  }
}

// the small diagnostics read back a few doubles through the pinned staging buffer
double PlaneEngine::read_scalars(int n, double *out) {
  LMW_LAUNCH_CHECK();
  LMW_CUDA(cudaMemcpyAsync(stage.p, diag.p, n * sizeof(double), cudaMemcpyDeviceToHost, stream));
  LMW_CUDA(cudaStreamSynchronize(stream));
  for (int k = 0; k < n; k++) out[k] = stage.p[k];
  return out[0];
}

// cpp/plane.cpp:245-264 (h_at, u_at, v_at); any finite point is read in bounds (periodic x, clamped rows)
double PlaneEngine::probe(int kind, double x, double y) {
  if (kind < 0 || kind > 2) throw InvalidArgument("field must be 0 (h), 1 (u) or 2 (v)");
  if (!std::isfinite(x) || !std::isfinite(y)) throw InvalidArgument("point outside the domain");
  plane_point<<<1, 1, 0, stream>>>(make_dev(p, *div), h0.p, u0.p, v0.p, kind, x, y, 0, 0, diag.p);
  g_launches += 1;
  double r;
  return read_scalars(1, &r);
}

// cpp/plane.cpp:220-226; corners i in 0..nx, j in 0..ny
double PlaneEngine::zeta_at_corner(int i, int j) {
  if (i < 0 || i > p.nx || j < 0 || j > p.ny) throw InvalidArgument("corner outside the grid");
  plane_point<<<1, 1, 0, stream>>>(make_dev(p, *div), h0.p, u0.p, v0.p, 3, 0.0, 0.0, i, j, diag.p);
  g_launches += 1;
  double r;
  return read_scalars(1, &r);
}

void PlaneEngine::row_harmonic(int kind, int m, int j, double shift, double *re, double *im) {
  const double *f = kind == 0 ? h0.p : kind == 1 ? u0.p : v0.p;
  plane_row_harmonics<<<1, HARM_THREADS, 0, stream>>>(f, p.nx, j, m, shift, reinterpret_cast<double2 *>(diag.p));
  g_launches += 1;
  double c[2];
  read_scalars(2, c);
  *re = c[0];
  *im = c[1];
}

// crest x of f ~ cos(2 pi m x / lx + ph), in [0, lx/m) (cpp/plane.cpp:284-289)
static double crest_x(const PlaneConfig &p, int m, double re, double im) {
  const double ph = std::atan2(im, re);
  double x = -ph / (2 * kPiPlane * m) * p.lx;
  const double per = p.lx / m;
  x = std::fmod(x, per);
  return x < 0 ? x + per : x;
}

// cpp/plane.cpp:271-277
double PlaneEngine::zonal_amplitude(int m, int j) {
  if (m < 1 || m >= p.nx / 2 || j < 0 || j >= p.ny) throw InvalidArgument("zonal harmonic or row out of range");
  double re, im;
  row_harmonic(0, m, j, 0.5, &re, &im);
  return 2 * std::hypot(re, im);
}

// cpp/plane.cpp:278-290
double PlaneEngine::zonal_crest(int m, int j) {
  if (m < 1 || m >= p.nx / 2 || j < 0 || j >= p.ny) throw InvalidArgument("zonal harmonic or row out of range");
  double re, im;
  row_harmonic(0, m, j, 0.5, &re, &im);
  return crest_x(p, m, re, im);
}

// cpp/plane.cpp:300-310 (v rows 1..ny-1)
double PlaneEngine::v_zonal_crest(int m, int j) {
  if (m < 1 || m >= p.nx / 2 || j < 1 || j >= p.ny) throw InvalidArgument("zonal harmonic or v row out of range");
  double re, im;
  row_harmonic(2, m, j, 0.5, &re, &im);
  return crest_x(p, m, re, im);
}

// cpp/plane.cpp:291-299: every u row and the interior v rows, one CTA per row, summed on the device
double PlaneEngine::harmonic_energy(int m) {
  if (m < 1 || m >= p.nx / 2) throw InvalidArgument("zonal harmonic out of range");
  double2 *c = reinterpret_cast<double2 *>(diag.p) + 1;
  plane_row_harmonics<<<p.ny, HARM_THREADS, 0, stream>>>(u0.p, p.nx, 0, m, 0.0, c);
  plane_row_harmonics<<<p.ny - 1, HARM_THREADS, 0, stream>>>(v0.p, p.nx, 1, m, 0.5, c + p.ny);
  plane_harmonic_energy_sum<<<1, 1, 0, stream>>>(c, 2 * p.ny - 1, p.ny, diag.p);
  g_launches += 3;
  double r;
  return read_scalars(1, &r);
}

// ------------------------------------------------------------------------------------------------ text writers
// cpp/main.cpp:464-478: per cell x y h uc vc zeta (zeta the mean of the four corner vorticities), a blank line after
// each row; the fields come back once and the host forms the cell values in the reference's order
void PlaneEngine::save_csv(const std::string &path) {
  const int nx = p.nx, ny = p.ny;
  std::vector<double> h(ncell()), u(ncell()), v(nvpt());
  get(h.data(), u.data(), v.data());
  const double dxx = dx(), dyy = dy();
  auto zc = [&](int i, int j) {  // cpp/plane.cpp:220-226
    const int im = (i + nx - 1) % nx;
    const double dvdx = (v[static_cast<size_t>(j) * nx + i % nx] - v[static_cast<size_t>(j) * nx + im]) / dxx;
    const double uj = j < ny ? u[static_cast<size_t>(j) * nx + i % nx] : u[static_cast<size_t>(ny - 1) * nx + i % nx];
    const double ujm = j > 0 ? u[static_cast<size_t>(j - 1) * nx + i % nx] : u[i % nx];
    return dvdx - (uj - ujm) / dyy;
  };
  std::string t;
  t.reserve(ncell() * 80);
  for (int j = 0; j < ny; j++) {
    for (int i = 0; i < nx; i++) {
      const size_t e = static_cast<size_t>(j) * nx + i;
      const double uc = 0.5 * (u[e] + u[static_cast<size_t>(j) * nx + (i + 1) % nx]), vc = 0.5 * (v[e] + v[e + nx]);
      const double z = 0.25 * (zc(i, j) + zc(i + 1, j) + zc(i, j + 1) + zc(i + 1, j + 1));
      t += fmt_g((i + 0.5) * dxx) + " " + fmt_g((j + 0.5) * dyy) + " " + fmt_g(h[e]) + " " + fmt_g(uc) + " " + fmt_g(vc) + " " + fmt_g(z) + "\n";
    }
    t += "\n";
  }
  write_text(path, t, "Plane.save_csv");
}

// cpp/main.cpp:480-487: x and h along row j
void PlaneEngine::save_row(int j, const std::string &path) {
  if (j < 0 || j >= p.ny) throw InvalidArgument("Plane.save_row: row outside the grid");
  std::vector<double> h(ncell());
  get(h.data(), nullptr, nullptr);
  std::string t;
  for (int i = 0; i < p.nx; i++) t += fmt_g((i + 0.5) * dx()) + " " + fmt_g(h[static_cast<size_t>(j) * p.nx + i]) + "\n";
  write_text(path, t, "Plane.save_row");
}

// cpp/main.cpp:488-494: y and h along column i
void PlaneEngine::save_column(int i, const std::string &path) {
  if (i < 0 || i >= p.nx) throw InvalidArgument("Plane.save_column: column outside the grid");
  std::vector<double> h(ncell());
  get(h.data(), nullptr, nullptr);
  std::string t;
  for (int j = 0; j < p.ny; j++) t += fmt_g((j + 0.5) * dy()) + " " + fmt_g(h[static_cast<size_t>(j) * p.nx + i]) + "\n";
  write_text(path, t, "Plane.save_column");
}

// cpp/plane.cpp:191-243: mean_depth, energy, max_speed, pv_anomaly_rms
void PlaneEngine::diagnostics(double *out) {
  Reduce r;
  reduce(r);
  const double N = static_cast<double>(ncell());
  out[0] = r.sum[0] / N;
  out[1] = r.sum[3] / N;
  out[2] = r.max[0];
  out[3] = std::sqrt(r.sum[4] / static_cast<double>(static_cast<size_t>(p.nx) * (p.ny - 1)));
}

}  // namespace lmw
