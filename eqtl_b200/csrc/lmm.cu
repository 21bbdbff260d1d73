// LMM path: eigenbasis, spectral rotation (K3), batched REML (K7) and the
// trans/gw LMM scan (K5).
//
// Restates src/model_lmm.cpp and src/scan_trans_lmm.cpp:82-251 on the
// shared-keep path:
//   basis     K = Q diag(lambda) Q', lambda clipped at 0 (make_lmm_basis,
//             src/model_lmm.cpp:106-113) - cuSOLVER syevd, or a basis the
//             caller supplies;
//   rotate    Gt = Q' (g - mean) for every kept SNP on the tensor cores
//             (FP16 hi/lo x hi/lo), written once as FP16 hi/lo pairs of Gt
//             and Gt^2 (the SNP-side operands of the scan);
//   REML      per gene: y~ = Q'y, X~ = Q'X, delta by the reference's grid /
//             golden-section / Newton search on reml_negll
//             (src/model_lmm.cpp:10-86), then dinv, A00, chi0, rss_null
//             (prep_lmm, :124-153) - one CTA per gene, FP64;
//   scan      per (gene, SNP) the bordered-Schur Wald test
//             (src/scan_trans_lmm.cpp:11-40) from three contractions
//               NUM = Gt . (w o r~)      (= yg - a'chi0, r~ = y~ - X~ chi0)
//               a_k = Gt . (w o X~_k)
//               gg  = Gt^2 . w
//             S = gg - a' A00^-1 a, t^2 = df r/(1-r), r = NUM^2/(S rss_null);
//   refine    candidates and each gene's best recomputed in FP64 from raw
//             dosages rotated by cuBLAS DGEMM.
#include <cublas_v2.h>
#include <cusolverDn.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <limits>
#include <memory>
#include <type_traits>

#include "internal.hpp"
#include "scan_host.hpp"
#include "simt_tile.cuh"
#include "tstat.hpp"

namespace eqtl {
namespace dev {

constexpr int kMaxPLmm = 32;
static_assert(kMaxPLmm + 2 <= kMaxAcc, "the grouped LMM scan needs p + 2 accumulators");
static_assert(sizeof(Workspace::ops_hi) / sizeof(Workspace::ops_hi[0]) >= static_cast<size_t>(kMaxAcc),
              "one gene-side operand buffer per accumulator");

// ----------------------------------------------------------- rotation
struct RotEpiParams {
  int64_t m;      // SNPs
  int k_pad;      // columns of the output rows; those past the eigenvectors are zero
  float unscale;  // accumulator -> Gt
  float s1, s2;   // output scales of Gt and Gt^2
  __half *gt_hi, *gt_lo, *gt2_hi, *gt2_lo;
};

struct RotEpi {
  static constexpr bool kGrouped = false;
  using Params = RotEpiParams;
  const Params& P;
  int row = 0;
  int64_t col0 = 0;
  static constexpr int kSmemBytes = 0;
  __device__ RotEpi(const Params& p, const TileShape&, uint8_t*) : P(p) {}
  __device__ void init(int, int) {}
  __device__ void begin_tile(int r, int64_t c0) {
    row = r;
    col0 = c0;
  }
  template <int NACC>
  __device__ void chunk(int c, const float (&v)[NACC][16]) {
    if (row >= P.k_pad) return;  // rows n .. k_pad are zero, as the tile's are
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int64_t s = col0 + c + j;
      if (s >= P.m) break;
      const float g = v[0][j] * P.unscale;
      const float a = g * P.s1;
      const float b = g * g * P.s2;
      const __half ah = __float2half_rn(a), bh = __float2half_rn(b);
      const int64_t idx = s * P.k_pad + row;
      P.gt_hi[idx] = ah;
      P.gt_lo[idx] = __float2half_rn(a - __half2float(ah));
      P.gt2_hi[idx] = bh;
      P.gt2_lo[idx] = __float2half_rn(b - __half2float(bh));
    }
  }
  __device__ void end_tile() {}
  __device__ void finish() {}
};

// Qt operand: row j = eigenvector j (column j of column-major Q) * 2^10.
// Q' split into hi + lo rows of T (FP16, or BF16 for the split-BF16 form,
// whose genotype operand is BF16 too)
template <class T>
__global__ void q_split_kernel(const double* __restrict__ Q, int n, int k_pad, T* hi, T* lo) {
  const int j = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k_pad; i += gridDim.x * blockDim.x) {
    const double v = i < n ? Q[static_cast<int64_t>(j) * n + i] * 1024.0 : 0.0;
    if constexpr (std::is_same_v<T, __half>) {
      const __half h = __double2half(v);
      hi[static_cast<int64_t>(j) * k_pad + i] = h;
      lo[static_cast<int64_t>(j) * k_pad + i] = __double2half(v - static_cast<double>(__half2float(h)));
    } else {
      const __nv_bfloat16 h = __double2bfloat16(v);
      hi[static_cast<int64_t>(j) * k_pad + i] = h;
      lo[static_cast<int64_t>(j) * k_pad + i] = __double2bfloat16(v - static_cast<double>(__bfloat162float(h)));
    }
  }
}

// --------------------------------------------------------------- REML
// Packed upper-triangle index of (a, b), a <= b.
__device__ __forceinline__ int tri(int a, int b, int p) { return a * p - a * (a - 1) / 2 + (b - a); }

// Solves A x = b for SPD A (p x p, row-major, Cholesky); returns false if not PD.
__device__ bool chol_solve(const double* A, const double* b, double* x, double* logdet, int p, double* L) {
  for (int j = 0; j < p; ++j) {
    double d = A[j * p + j];
    for (int k = 0; k < j; ++k) d -= L[j * p + k] * L[j * p + k];
    if (!(d > 0)) return false;
    L[j * p + j] = sqrt(d);
    for (int i = j + 1; i < p; ++i) {
      double s = A[i * p + j];
      for (int k = 0; k < j; ++k) s -= L[i * p + k] * L[j * p + k];
      L[i * p + j] = s / L[j * p + j];
    }
  }
  double ld = 0;
  for (int j = 0; j < p; ++j) ld += 2.0 * log(L[j * p + j]);
  *logdet = ld;
  if (b) {
    double y[kMaxPLmm];
    for (int i = 0; i < p; ++i) {
      double s = b[i];
      for (int k = 0; k < i; ++k) s -= L[i * p + k] * y[k];
      y[i] = s / L[i * p + i];
    }
    for (int i = p - 1; i >= 0; --i) {
      double s = y[i];
      for (int k = i + 1; k < p; ++k) s -= L[k * p + i] * x[k];
      x[i] = s / L[i * p + i];
    }
  }
  return true;
}

// prep_lmm caches (src/model_lmm.cpp:124-153) from A = X~'DX~ (p x p,
// row-major), b = X~'Dy~ and y~'Dy~ at the chosen delta; one thread. Besides
// chi0, A^-1 and rss, the lower Cholesky factor of A (row-major, zeros when A
// is not positive definite) for the FP64 pair statistics.
__device__ void reml_caches(double* A, const double* b, double y_dy, int p, int g, double* L, double* e,
                            double* x, double* chi0_out, double* ainv_out, double* rss_out, double* a00L_out) {
  double chi0[kMaxPLmm];
  double ld;
  const bool ok = chol_solve(A, b, chi0, &ld, p, L);
  double rss = y_dy;
  for (int i = 0; i < p; ++i)
    for (int j = 0; j < p; ++j)
      a00L_out[(static_cast<int64_t>(g) * p + i) * p + j] = ok && j <= i ? L[i * p + j] : 0.0;
  if (ok) {
    for (int k = 0; k < p; ++k) rss -= b[k] * chi0[k];
    if (rss < 0) rss = 0;
    for (int c = 0; c < p; ++c) {  // A00^-1 column by column
      for (int i = 0; i < p; ++i) e[i] = (i == c) ? 1.0 : 0.0;
      double dummy;
      chol_solve(A, e, x, &dummy, p, L);
      for (int i = 0; i < p; ++i) ainv_out[(static_cast<int64_t>(g) * p + i) * p + c] = x[i];
    }
  } else {
    for (int k = 0; k < p; ++k) chi0[k] = 0;
    for (int i = 0; i < p * p; ++i) ainv_out[static_cast<int64_t>(g) * p * p + i] = 0;
  }
  rss_out[g] = rss;
  for (int k = 0; k < p; ++k) chi0_out[static_cast<int64_t>(g) * p + k] = chi0[k];
}

// Grid of the search: f(1.0), then 1e-5 * 2^k for k = 0..33 (the loop dd <= 1e5,
// dd *= 2); 1e-5 doubled k times is exact, so this is the reference's dd sequence.
constexpr int kRbGridN = 35;
__device__ __forceinline__ double rb_grid_delta(int j) { return j == 0 ? 1.0 : ldexp(1e-5, j - 1); }

// ---- REML -loglik (src/model_lmm.cpp:10-37) for P <= 3 covariate columns,
// evaluated by one warp: each lane sums log v, w y^2, w x_a x_b and w y x_a over
// its samples in registers, and xor-shuffle reductions give every lane the same
// totals (IEEE addition is commutative), so there is no shared memory and no
// block barrier. tot = [sum log v, y'Dy, X'DX packed (a <= b), X'Dy].
template <int P>
struct RemlSums {
  static constexpr int NQ = P * (P + 1) / 2, V = 2 + NQ + P;
  double acc[V], prod = 1.0;
  int nprod = 0;
  __device__ __forceinline__ RemlSums() {
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = 0.0;
  }
  // weight of a sample, and its log v: the sum of logs as the log of products of
  // up to eight factors; every factor lies in [1e-12, 1e36] (larger ones take
  // their own log), so a product stays within [1e-96, 1e288]
  __device__ __forceinline__ double weight(double delta, double lam) {
    double v = delta * lam + 1.0;
    if (v < 1e-12) v = 1e-12;
    if (v <= 1e36) {
      prod *= v;
      if (++nprod == 8) {
        acc[0] += log(prod);
        prod = 1.0;
        nprod = 0;
      }
    } else {
      acc[0] += log(v);
    }
    return 1.0 / v;
  }
  __device__ __forceinline__ void add_x(double w, const double (&x)[P]) {
#pragma unroll
    for (int a = 0; a < P; ++a)
#pragma unroll
      for (int b = a; b < P; ++b) acc[2 + a * P - a * (a - 1) / 2 + (b - a)] += w * x[a] * x[b];
  }
  __device__ __forceinline__ void add_y(double w, double y, const double (&x)[P]) {
    acc[1] += w * y * y;
#pragma unroll
    for (int a = 0; a < P; ++a) acc[2 + NQ + a] += w * y * x[a];
  }
  __device__ __forceinline__ void end() {
    acc[0] += log(prod);
#pragma unroll
    for (int q = 0; q < V; ++q)
#pragma unroll
      for (int o = 16; o; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
  }
};

// -loglik from the totals: Cholesky of X'DX; q = y'Dy - b'(X'DX)^-1 b as
// y'Dy - |z|^2 with L z = b. No shuffles: lanes may hold different totals.
template <int P>
__device__ __forceinline__ double reml_ll(const double (&tot)[RemlSums<P>::V], int n) {
  constexpr int NQ = RemlSums<P>::NQ;
  double L[P][P];
  double logdet_x = 0.0;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    double d = tot[2 + j * P - j * (j - 1) / 2];
#pragma unroll
    for (int k = 0; k < j; ++k) d -= L[j][k] * L[j][k];
    if (!(d > 0)) return 1e300;
    L[j][j] = sqrt(d);
    logdet_x += 2.0 * log(L[j][j]);
#pragma unroll
    for (int i = j + 1; i < P; ++i) {
      double s = tot[2 + j * P - j * (j - 1) / 2 + (i - j)];
#pragma unroll
      for (int k = 0; k < j; ++k) s -= L[i][k] * L[j][k];
      L[i][j] = s / L[j][j];
    }
  }
  double q = tot[1];
  double z[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    double s = tot[2 + NQ + i];
#pragma unroll
    for (int k = 0; k < i; ++k) s -= L[i][k] * z[k];
    z[i] = s / L[i][i];
    q -= z[i] * z[i];
  }
  if (q <= 0) q = 1e-12;
  const double df = static_cast<double>(n - P);
  return 0.5 * (df * log(q / df) + tot[0] + logdet_x);
}

// The grid's deltas are the same for every gene: one warp per grid point keeps
// the weights w_k,i in Wg[i + n k] and the totals that y has no part in, sum log v
// and X'DX, in Gt[k][1 + NQ].
template <int P>
__global__ void reml_grid_kernel(const double* __restrict__ Xtil, const double* __restrict__ lam, int n,
                                 double* __restrict__ Wg, double* __restrict__ Gt) {
  const int k = blockIdx.x, lane = threadIdx.x;
  const double delta = rb_grid_delta(k);
  RemlSums<P> s;
  for (int i = lane; i < n; i += 32) {
    const double w = s.weight(delta, lam[i]);
    double x[P];
#pragma unroll
    for (int a = 0; a < P; ++a) x[a] = Xtil[static_cast<int64_t>(a) * n + i];
    s.add_x(w, x);
    Wg[static_cast<int64_t>(k) * n + i] = w;
  }
  s.end();
  if (lane == 0) {
    constexpr int NG = 1 + RemlSums<P>::NQ;
    Gt[k * NG] = s.acc[0];
#pragma unroll
    for (int q = 1; q < NG; ++q) Gt[k * NG + q] = s.acc[1 + q];
  }
}

// One warp per gene for P <= 3 (intercept and a few covariates): optimize_delta
// (src/model_lmm.cpp:39-86: grid 1e-5..1e5 x2 and 1.0, 40 golden-section steps on
// [best/4, best*4] clipped to [1e-8, 1e6], then up to 8 Newton steps on central
// differences) and the prep_lmm caches (:124-153).
//
// Bound by FP64 issue: ~24 operations a sample and delta, of which the weight's
// division and log are 15. The grid's weights come from reml_grid_kernel (four
// operations a sample remain), five grid points share the loads of y and x, as do
// the two deltas of a golden-section or Newton step; the -logliks of 32 grid
// points, or of the step's two deltas, are then computed in different lanes of
// one pass. Every sum keeps its order. n = 2000, 10,000 genes, P = 1: 6.7 ->
// 3.9 ms; n = 1201, 1,503 genes, P = 2: 1.93 -> 0.88 ms.
constexpr int kRemlWarpP = 3;
constexpr int kRemlThreads = 64;  // two genes a block: an even last wave for a few thousand genes
constexpr int kRemlGridStep = 5;  // grid points per pass over the samples
template <int P>
__global__ void __launch_bounds__(kRemlThreads) reml_warp_kernel(
    const double* __restrict__ Ytil, const double* __restrict__ Xtil, const double* __restrict__ lam, int n, int G,
    const double* __restrict__ Wg, const double* __restrict__ Gt, double* delta_out, double* chi0_out,
    double* ainv_out, double* rss_out, double* a00L_out) {
  constexpr int NQ = RemlSums<P>::NQ, V = RemlSums<P>::V, NG = 1 + NQ;
  static_assert(kRbGridN % kRemlGridStep == 0 && kRbGridN <= 64, "grid passes");
  const int g = blockIdx.x * (kRemlThreads >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (g >= G) return;  // whole warps only: no block barrier follows
  const double* yt = Ytil + static_cast<int64_t>(g) * n;
  auto load_x = [&](int i, double (&x)[P]) {
#pragma unroll
    for (int a = 0; a < P; ++a) x[a] = Xtil[static_cast<int64_t>(a) * n + i];
  };
  auto f = [&](double d, RemlSums<P>& s) {
    for (int i = lane; i < n; i += 32) {
      const double w = s.weight(d, lam[i]), y = yt[i];
      double x[P];
      load_x(i, x);
      s.add_x(w, x);
      s.add_y(w, y, x);
    }
    s.end();
    return reml_ll<P>(s.acc, n);
  };
  auto f1 = [&](double d) {
    RemlSums<P> s;
    return f(d, s);
  };
  auto f2 = [&](double d0, double d1, double& r0, double& r1) {
    RemlSums<P> s0, s1;
    for (int i = lane; i < n; i += 32) {
      const double l = lam[i], y = yt[i];
      double x[P];
      load_x(i, x);
      const double w0 = s0.weight(d0, l), w1 = s1.weight(d1, l);
      s0.add_x(w0, x);
      s0.add_y(w0, y, x);
      s1.add_x(w1, x);
      s1.add_y(w1, y, x);
    }
    s0.end();
    s1.end();
#pragma unroll
    for (int q = 0; q < V; ++q) s0.acc[q] = lane < 16 ? s0.acc[q] : s1.acc[q];
    const double r = reml_ll<P>(s0.acc, n);
    r0 = __shfl_sync(0xffffffffu, r, 0);
    r1 = __shfl_sync(0xffffffffu, r, 16);
  };

  double d = 1.0;
  if (n - P > 0) {
    // grid: lane l takes the totals of points l and 32 + l
    double ty[2][1 + P];
#pragma unroll 1
    for (int k0 = 0; k0 < kRbGridN; k0 += kRemlGridStep) {
      double acc[kRemlGridStep][1 + P];
#pragma unroll
      for (int j = 0; j < kRemlGridStep; ++j)
#pragma unroll
        for (int q = 0; q <= P; ++q) acc[j][q] = 0.0;
      const double* wk = Wg + static_cast<int64_t>(k0) * n;
      for (int i = lane; i < n; i += 32) {
        const double y = yt[i];
        double x[P];
        load_x(i, x);
#pragma unroll
        for (int j = 0; j < kRemlGridStep; ++j) {
          const double w = wk[static_cast<int64_t>(j) * n + i];
          acc[j][0] += w * y * y;
#pragma unroll
          for (int a = 0; a < P; ++a) acc[j][1 + a] += w * y * x[a];
        }
      }
#pragma unroll
      for (int j = 0; j < kRemlGridStep; ++j) {
#pragma unroll
        for (int q = 0; q <= P; ++q) {
#pragma unroll
          for (int o = 16; o; o >>= 1) acc[j][q] += __shfl_xor_sync(0xffffffffu, acc[j][q], o);
          if (lane == ((k0 + j) & 31)) {
            if (k0 + j < 32) ty[0][q] = acc[j][q];
            else ty[1][q] = acc[j][q];
          }
        }
      }
    }
    double ll[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = h * 32 + lane;
      ll[h] = CUDART_NAN;  // no point: never the smallest
      if (k < kRbGridN) {
        double tot[V];
        tot[0] = Gt[k * NG];
        tot[1] = ty[h][0];
#pragma unroll
        for (int q = 1; q < NG; ++q) tot[1 + q] = Gt[k * NG + q];
#pragma unroll
        for (int a = 0; a < P; ++a) tot[2 + NQ + a] = ty[h][1 + a];
        ll[h] = reml_ll<P>(tot, n);
      }
    }
    // the first of the smallest values; where f(1.0) is NaN nothing is below it
    int best = lane;
    double bl = ll[0];
    if (ll[1] < bl || (isnan(bl) && !isnan(ll[1]))) {
      bl = ll[1];
      best = 32 + lane;
    }
    const double ll0 = __shfl_sync(0xffffffffu, ll[0], 0);
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const double v = __shfl_xor_sync(0xffffffffu, bl, o);
      const int k = __shfl_xor_sync(0xffffffffu, best, o);
      if (v < bl || (v == bl && k < best) || (isnan(bl) && !isnan(v))) {
        bl = v;
        best = k;
      }
    }
    const double best_d = rb_grid_delta(isnan(ll0) ? 0 : best);
    double lo = best_d / 4.0, hi = best_d * 4.0;
    if (lo < 1e-8) lo = 1e-8;
    if (hi > 1e6) hi = 1e6;
    const double phi = (1.0 + sqrt(5.0)) / 2.0;
    for (int it = 0; it < 40; ++it) {
      const double m1 = hi - (hi - lo) / phi;
      const double m2 = lo + (hi - lo) / phi;
      double v1, v2;
      f2(m1, m2, v1, v2);
      if (v1 < v2) hi = m2;
      else lo = m1;
    }
    d = 0.5 * (lo + hi);
    double cur = f1(d);
    for (int it = 0; it < 8; ++it) {
      const double h = fmax(d * 1e-4, 1e-9);
      double fm, fp;
      f2(d - h, d + h, fm, fp);
      const double g1 = (fp - fm) / (2.0 * h);
      const double g2 = (fp - 2.0 * cur + fm) / (h * h);
      if (!(g2 > 1e-12)) break;
      const double step = g1 / g2;
      const double dn = d - step;
      if (!(dn > 1e-8 && dn < 1e6)) break;
      const double vn = f1(dn);
      if (!(vn < cur)) break;
      d = dn;
      cur = vn;
      if (fabs(step) < d * 1e-8) break;
    }
  }
  RemlSums<P> s;
  f(d, s);
  if (lane == 0) {
    double A[P * P], L[P * P], e[P], x[P];
    for (int a = 0; a < P; ++a)
      for (int b = a; b < P; ++b) A[a * P + b] = A[b * P + a] = s.acc[2 + a * P - a * (a - 1) / 2 + (b - a)];
    delta_out[g] = d;
    reml_caches(A, s.acc + 2 + NQ, s.acc[1], P, g, L, e, x, chi0_out, ainv_out, rss_out, a00L_out);
  }
}

// ------------------------------------------- batched REML (p > kRemlWarpP)
// The same schedule and -loglik for many columns in lockstep. Each round
// evaluates up to two deltas per column (slot s = slot * C + column); the
// sums over the n samples run as FP64 GEMMs shared by all columns,
//   A[q, s] = sum_i P[q, i] W[i, s]     P[q, i] = x~_ai x~_bi (q = tri(a, b))
//   b[a, s] = sum_i x~_ai (W o Y)[i, s]
// with W[i, s] = 1 / max(delta_s lambda_i + 1, 1e-12), and groups of 8, 16 or 32
// lanes factorise a column's sums and advance its search (golden section, Newton)
// between rounds; the grid phase, whose deltas every column shares, runs once before
// them.
enum : int { kRbGolden = 1, kRbCentre, kRbNewtonPair, kRbNewtonStep, kRbFinal };
constexpr int kRbMaxRounds = 40 + 1 + 2 * 8 + 1;  // golden, centre, Newton, final

struct RemlBatchState {
  int phase, k;
  double best_d, best_ll, lo, hi, d, cur, h, step, dn;
};

__device__ void rb_propose(const RemlBatchState& s, double& d0, double& d1) {
  d0 = d1 = CUDART_NAN;
  switch (s.phase) {
    case kRbGolden: {
      const double phi = (1.0 + sqrt(5.0)) / 2.0;
      d0 = s.hi - (s.hi - s.lo) / phi;
      d1 = s.lo + (s.hi - s.lo) / phi;
      break;
    }
    case kRbCentre:
    case kRbFinal:
      d0 = s.d;
      break;
    case kRbNewtonPair:
      d0 = s.d - s.h;
      d1 = s.d + s.h;
      break;
    case kRbNewtonStep:
      d0 = s.dn;
      break;
    default:
      break;
  }
}

// P[q + nq i] = x~_ai x~_bi
__global__ void rb_pairs_kernel(const double* __restrict__ Xtil, int n, int p, double* P) {
  const int nq = p * (p + 1) / 2;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < static_cast<int64_t>(nq) * n;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int q = static_cast<int>(t % nq);
    const int i = static_cast<int>(t / nq);
    int a = 0;
    while (tri(a, p - 1, p) < q) ++a;
    const int b = a + (q - tri(a, a, p));
    P[t] = Xtil[static_cast<int64_t>(a) * n + i] * Xtil[static_cast<int64_t>(b) * n + i];
  }
}

// ---- grid phase, shared by all columns: the 35 grid deltas are the same for
// every column, so D_k, X~'D_k X~ (and its Cholesky factor) and sum log v
// are computed once; per column only X~'D_k y and y'D_k y remain (GEMMs).
// Wg[i + n k] = w_k,i, Xw[i + n (k p + a)] = w_k,i x~_ai, ldD[k] = sum_i log v_k,i.
__global__ void rb_grid_weights_kernel(const double* __restrict__ Xtil, const double* __restrict__ lam, int n,
                                       int p, double* Wg, double* Xw, double* ldD) {
  const int k = blockIdx.x;  // grid point
  const double delta = rb_grid_delta(k);
  const int lane = threadIdx.x & 31;
  double acc = 0.0, prod = 1.0;
  int nprod = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double v = delta * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    const double w = 1.0 / v;
    Wg[i + static_cast<int64_t>(n) * k] = w;
    for (int a = 0; a < p; ++a)
      Xw[i + static_cast<int64_t>(n) * (k * p + a)] = w * Xtil[static_cast<int64_t>(a) * n + i];
    if (v <= 1e36) {
      prod *= v;
      if (++nprod == 8) {
        acc += log(prod);
        prod = 1.0;
        nprod = 0;
      }
    } else {
      acc += log(v);
    }
  }
  acc += log(prod);
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ double red[32];
  if (lane == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) t += red[w];
    ldD[k] = t;
  }
}

// ---- one p x p factorisation per group of GW lanes (GW = 8, 16 or 32, p <= GW)
// One thread per column used to factorise and solve alone: at p = 16 that is
// a chain of ~1,500 dependent FP64 operations on local memory, 325 us a round
// whatever the number of columns (72 % of a 500-column cis scan's device
// time). Here lane i of the group holds row i in registers and the updates of
// a step run across the lanes; every element still sees the same operations
// in the same order (column k of the factor is subtracted before column
// k + 1), so each factor, solution and -loglik keeps its bits.
// Measured at n = 1000, p = 16: the null fits of 500 columns 18.3 -> 3.7 ms, of
// 8,000 columns 39.7 -> 22.3 ms (this kernel 55 us a round there).
template <int GW>
__device__ __forceinline__ double rb_shfl(double v, int src) {
  return __shfl_sync(0xffffffffu, v, src, GW);
}

// Lower Cholesky factor of the SPD matrix whose packed upper triangle is A
// (tri order) and, in the same sweep, the forward solve L y = b (b == null:
// not wanted): on return row[c] = L[gl][c] (c <= gl) in lane gl, diag = L[gl][gl],
// y = y[gl], *logdet = log det A. Lanes gl >= p carry an identity. Returns
// false (to the whole group) where a pivot is not positive; the values are
// then meaningless. Every lane of the warp takes part.
template <int GW>
__device__ __forceinline__ bool rb_factor(const double* __restrict__ A, const double* __restrict__ b, int p, int gl,
                                          double (&row)[GW], double& diag, double& y, double* logdet) {
#pragma unroll
  for (int c = 0; c < GW; ++c) row[c] = gl < p && c <= gl ? A[tri(c, gl, p)] : (c == gl ? 1.0 : 0.0);
  y = b && gl < p ? b[gl] : 0.0;
  diag = 1.0;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < GW; ++j) {
    if (j < p) {  // uniform across the launch
      const double d = rb_shfl<GW>(row[j], j);
      ok = ok && d > 0;
      const double ljj = sqrt(d);
      const double lij = gl == j ? ljj : row[j] / ljj;
      const double yj = rb_shfl<GW>(y, j) / ljj;
      row[j] = lij;
      if (gl == j) {
        diag = ljj;
        y = yj;
      }
      if (gl > j) y = fma(-lij, yj, y);
#pragma unroll
      for (int c = j + 1; c < GW; ++c)
        if (c < p) {
          const double lcj = rb_shfl<GW>(lij, c);
          if (gl >= c) row[c] = fma(-lij, lcj, row[c]);
        }
    }
  }
  const double lg = log(diag);
  double ld = 0.0;
#pragma unroll
  for (int j = 0; j < GW; ++j)
    if (j < p) ld += 2.0 * rb_shfl<GW>(lg, j);
  *logdet = ld;
  return ok;
}

// Lg[k] = Cholesky factor of X~'D_k X~ (row-major, lower), ldx[k] its log
// determinant, or ldx[k] = NaN when it is not positive definite. One group of
// GW lanes per grid point.
template <int GW>
__global__ void __launch_bounds__(128) rb_grid_chol_kernel(const double* __restrict__ Ag, int p, double* Lg,
                                                           double* ldx) {
  const int k0 = (blockIdx.x * blockDim.x + threadIdx.x) / GW;
  const int gl = threadIdx.x % GW;
  const int k = min(k0, kRbGridN - 1);  // spare groups repeat the last point and write nothing
  const int nq = p * (p + 1) / 2;
  double row[GW], diag, y, ld;
  const bool ok = rb_factor<GW>(Ag + static_cast<int64_t>(k) * nq, nullptr, p, gl, row, diag, y, &ld);
  if (k0 >= kRbGridN) return;
  double* L = Lg + static_cast<int64_t>(k) * p * p;
  if (gl < p) {
#pragma unroll
    for (int c = 0; c < GW; ++c)
      if (c <= gl) L[gl * p + c] = row[c];
  }
  if (gl == 0) ldx[k] = ok ? ld : CUDART_NAN;
}

// -loglik of every column at grid point k = blockIdx.y into V[k C + c] (one
// thread per column and grid point: the 35 forward solves of a column used to
// run one after the other in one thread, 514 us at 500 columns; the factor is
// read from shared memory).
// Bg[(k p + a) + 35 p c] = x~_a' D_k y_c, Yg[k + 35 c] = y_c' D_k y_c.
template <int GW>
__global__ void __launch_bounds__(128)
    rb_grid_eval_kernel(int C, int p, int df, const double* __restrict__ Lg, const double* __restrict__ ldx,
                        const double* __restrict__ ldD, const double* __restrict__ Bg,
                        const double* __restrict__ Yg, double* V) {
  __shared__ double L[GW * GW];
  const int k = blockIdx.y;
  for (int e = threadIdx.x; e < p * p; e += blockDim.x) L[e] = Lg[static_cast<int64_t>(k) * p * p + e];
  __syncthreads();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  double v = 1e300;
  const double lx = ldx[k];
  if (lx == lx) {
    const double dfd = static_cast<double>(df);
    const double* b = Bg + static_cast<int64_t>(kRbGridN) * p * c + static_cast<int64_t>(k) * p;
    double z[GW];
    double q = Yg[k + static_cast<int64_t>(kRbGridN) * c];
#pragma unroll
    for (int i = 0; i < GW; ++i)
      if (i < p) {
        double t = b[i];
#pragma unroll
        for (int j = 0; j < i; ++j) t -= L[i * p + j] * z[j];
        z[i] = t / L[i * p + i];
        q -= z[i] * z[i];
      }
    if (q <= 0) q = 1e-12;
    v = 0.5 * (dfd * log(q / dfd) + ldD[k] + lx);
  }
  V[static_cast<int64_t>(k) * C + c] = v;
}

// Per column: the best of the 35 grid -logliks in the reference's order
// (f(1.0) first, strict <), then the golden-section bracket; proposes the
// first round.
__global__ void rb_grid_advance_kernel(int C, int df, const double* __restrict__ V, RemlBatchState* st, double* dlt) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  RemlBatchState s{};
  s.d = 1.0;
  if (df <= 0) {
    s.phase = kRbFinal;
  } else {
    for (int k = 0; k < kRbGridN; ++k) {
      const double v = V[static_cast<int64_t>(k) * C + c];
      if (k == 0) {
        s.best_ll = v;
        s.best_d = 1.0;
      } else if (v < s.best_ll) {
        s.best_ll = v;
        s.best_d = rb_grid_delta(k);
      }
    }
    s.lo = s.best_d / 4.0;
    s.hi = s.best_d * 4.0;
    if (s.lo < 1e-8) s.lo = 1e-8;
    if (s.hi > 1e6) s.hi = 1e6;
    s.phase = kRbGolden;
  }
  st[c] = s;
  rb_propose(s, dlt[c], dlt[C + c]);
}

// One warp per slot: W, W o y, sum log v (log of eight-factor products, as in
// RemlSums) and y'Dy. Slots with no delta (NaN) are skipped. Bound by the
// latency of the FP64 reciprocals and loads when the columns are few, so a
// lane takes eight of its samples per step, whose reciprocals overlap; the
// sums keep each lane's sample order.
__global__ void __launch_bounds__(256) rb_weights_kernel(const double* __restrict__ Ytil,
                                                         const double* __restrict__ lam, int n, int C,
                                                         const double* __restrict__ dlt, double* W, double* WY,
                                                         double* ld, double* ydy) {
  const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (s >= 2 * C) return;
  const double delta = dlt[s];
  if (!(delta == delta)) return;
  const double* y = Ytil + static_cast<int64_t>(s % C) * n;
  double* w_out = W + static_cast<int64_t>(s) * n;
  double* wy_out = WY + static_cast<int64_t>(s) * n;
  double acc_ld = 0.0, acc_y = 0.0, prod = 1.0;
  int nprod = 0;
  int i = lane;
  for (; i + 7 * 32 < n; i += 8 * 32) {
    double v[8], yi[8];
    bool in = nprod == 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      v[t] = delta * lam[i + 32 * t] + 1.0;
      yi[t] = y[i + 32 * t];
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      if (v[t] < 1e-12) v[t] = 1e-12;
      in = in && v[t] <= 1e36;
      const double w = 1.0 / v[t];
      w_out[i + 32 * t] = w;
      wy_out[i + 32 * t] = w * yi[t];
      acc_y += w * yi[t] * yi[t];
    }
    if (in) {  // eight factors of one product, whose log is due
#pragma unroll
      for (int t = 0; t < 8; ++t) prod *= v[t];
      acc_ld += log(prod);
      prod = 1.0;
      continue;
    }
    for (int t = 0; t < 8; ++t) {  // a factor above 1e36 takes its own log
      double u = delta * lam[i + 32 * t] + 1.0;
      if (u < 1e-12) u = 1e-12;
      if (u <= 1e36) {
        prod *= u;
        if (++nprod == 8) {
          acc_ld += log(prod);
          prod = 1.0;
          nprod = 0;
        }
      } else {
        acc_ld += log(u);
      }
    }
  }
  for (; i < n; i += 32) {
    double v = delta * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    const double w = 1.0 / v;
    if (v <= 1e36) {
      prod *= v;
      if (++nprod == 8) {
        acc_ld += log(prod);
        prod = 1.0;
        nprod = 0;
      }
    } else {
      acc_ld += log(v);
    }
    const double yi = y[i];
    w_out[i] = w;
    wy_out[i] = w * yi;
    acc_y += w * yi * yi;
  }
  acc_ld += log(prod);
  for (int o = 16; o; o >>= 1) {
    acc_ld += __shfl_xor_sync(0xffffffffu, acc_ld, o);
    acc_y += __shfl_xor_sync(0xffffffffu, acc_y, o);
  }
  if (lane == 0) {
    ld[s] = acc_ld;
    ydy[s] = acc_y;
  }
}

// L (row stride GW + 1) of this group in shared memory, and beta = (L L')^-1 b
// from y = L^-1 b: every lane of the group runs the same back substitution,
// each element's terms in increasing order, as chol_solve does.
template <int GW>
__device__ __forceinline__ void rb_back_solve(const double (&row)[GW], double y, int p, int gl, double* L,
                                              double (&beta)[GW]) {
#pragma unroll
  for (int c = 0; c < GW; ++c) L[gl * (GW + 1) + c] = row[c];
  __syncwarp();
#pragma unroll
  for (int i = GW - 1; i >= 0; --i) {
    const double yi = rb_shfl<GW>(y, i);
    beta[i] = 0.0;
    if (i < p) {
      double s = yi;
#pragma unroll
      for (int k = i + 1; k < GW; ++k)
        if (k < p) s -= L[k * (GW + 1) + i] * beta[k];
      beta[i] = s / L[i * (GW + 1) + i];
    }
  }
}

constexpr int kRbThreads = 128;

// Two groups of GW lanes per column, one per slot, evaluate the round's
// -logliks; one lane then advances the search exactly as reml_warp_kernel
// does and proposes the next round's deltas. A column whose search has ended
// keeps proposing its delta (kRbFinal) until every column's has: the caches are
// formed for all of them at once (rb_final_kernel). *active counts the
// columns still searching.
template <int GW>
__global__ void __launch_bounds__(kRbThreads)
    rb_advance_kernel(int C, int p, int df, const double* __restrict__ A, const double* __restrict__ B,
                      const double* __restrict__ ld, const double* __restrict__ ydy, RemlBatchState* st, double* dlt,
                      unsigned int* active) {
  constexpr int kGroups = kRbThreads / GW;
  __shared__ double Ls[kGroups * GW * (GW + 1)];
  __shared__ double val[kGroups];
  const int grp = threadIdx.x / GW, gl = threadIdx.x % GW;
  const int slot = grp & 1;
  const int c0 = blockIdx.x * (kGroups / 2) + (grp >> 1);
  const int c = min(c0, C - 1);  // spare groups repeat the last column and write nothing
  const int nq = p * (p + 1) / 2;
  const int si = slot * C + c;
  // a slot without a delta this round holds an earlier round's sums; its value
  // is not read
  const double* b = B + static_cast<int64_t>(si) * p;
  double row[GW], beta[GW], diag, y, logdet_x;
  const bool ok = rb_factor<GW>(A + static_cast<int64_t>(si) * nq, b, p, gl, row, diag, y, &logdet_x);
  rb_back_solve<GW>(row, y, p, gl, Ls + grp * GW * (GW + 1), beta);
  if (gl == 0) {
    double q = ydy[si];
#pragma unroll
    for (int k = 0; k < GW; ++k)
      if (k < p) q -= b[k] * beta[k];
    if (q <= 0) q = 1e-12;
    const double dfd = static_cast<double>(df);
    val[grp] = ok ? 0.5 * (dfd * log(q / dfd) + ld[si] + logdet_x) : 1e300;
  }
  __syncthreads();
  if (gl != 0 || slot != 0 || c0 >= C) return;
  RemlBatchState s = st[c];
  if (s.phase == kRbFinal) return;
  const double f0 = val[grp], f1 = val[grp + 1];
  switch (s.phase) {
    case kRbGolden: {
      const double phi = (1.0 + sqrt(5.0)) / 2.0;
      const double m1 = s.hi - (s.hi - s.lo) / phi;
      const double m2 = s.lo + (s.hi - s.lo) / phi;
      if (f0 < f1) s.hi = m2;
      else s.lo = m1;
      if (++s.k == 40) {
        s.d = 0.5 * (s.lo + s.hi);
        s.phase = kRbCentre;
      }
      break;
    }
    case kRbCentre:
      s.cur = f0;
      s.k = 0;
      s.h = fmax(s.d * 1e-4, 1e-9);
      s.phase = kRbNewtonPair;
      break;
    case kRbNewtonPair: {
      const double fm = f0;
      const double fp = f1;
      const double g1 = (fp - fm) / (2.0 * s.h);
      const double g2 = (fp - 2.0 * s.cur + fm) / (s.h * s.h);
      s.phase = kRbFinal;
      if (g2 > 1e-12) {
        s.step = g1 / g2;
        s.dn = s.d - s.step;
        if (s.dn > 1e-8 && s.dn < 1e6) s.phase = kRbNewtonStep;
      }
      break;
    }
    case kRbNewtonStep: {
      const double vn = f0;
      s.phase = kRbFinal;
      if (vn < s.cur) {
        s.d = s.dn;
        s.cur = vn;
        if (!(fabs(s.step) < s.d * 1e-8) && ++s.k < 8) {
          s.h = fmax(s.d * 1e-4, 1e-9);
          s.phase = kRbNewtonPair;
        }
      }
      break;
    }
    default:
      break;
  }
  st[c] = s;
  rb_propose(s, dlt[c], dlt[C + c]);
  if (s.phase != kRbFinal) atomicAdd(active, 1u);
}

// After the last round, whose slot 0 holds every column's sums at its final
// delta: delta and the prep_lmm caches (reml_caches) with one group of GW lanes
// per column; lane k solves column k of A00^-1.
template <int GW>
__global__ void __launch_bounds__(kRbThreads)
    rb_final_kernel(int C, int g0, int p, const double* __restrict__ A, const double* __restrict__ B,
                    const double* __restrict__ ydy, const RemlBatchState* __restrict__ st, double* delta_out,
                    double* chi0_out, double* ainv_out, double* rss_out, double* a00L_out) {
  constexpr int kGroups = kRbThreads / GW;
  __shared__ double Ls[kGroups * GW * (GW + 1)];
  const int grp = threadIdx.x / GW, gl = threadIdx.x % GW;
  const int c0 = blockIdx.x * kGroups + grp;
  const int c = min(c0, C - 1);
  const int nq = p * (p + 1) / 2;
  const double* b = B + static_cast<int64_t>(c) * p;
  double row[GW], beta[GW], diag, y, logdet_x;
  const bool ok = rb_factor<GW>(A + static_cast<int64_t>(c) * nq, b, p, gl, row, diag, y, &logdet_x);
  double* L = Ls + grp * GW * (GW + 1);
  rb_back_solve<GW>(row, y, p, gl, L, beta);
  if (c0 >= C || gl >= p) return;
  const int64_t g = g0 + c;
  // column gl of A00^-1: L y = e_gl, then L' x = y
  double x[GW];
#pragma unroll
  for (int i = 0; i < GW; ++i) {
    x[i] = 0.0;
    if (i < p) {
      double s = i == gl ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < i; ++k) s -= L[i * (GW + 1) + k] * x[k];
      x[i] = s / L[i * (GW + 1) + i];
    }
  }
#pragma unroll
  for (int i = GW - 1; i >= 0; --i)
    if (i < p) {
      double s = x[i];
#pragma unroll
      for (int k = i + 1; k < GW; ++k)
        if (k < p) s -= L[k * (GW + 1) + i] * x[k];
      x[i] = s / L[i * (GW + 1) + i];
    }
#pragma unroll
  for (int i = 0; i < GW; ++i)
    if (i < p) {
      ainv_out[(g * p + i) * p + gl] = ok ? x[i] : 0.0;
      a00L_out[(g * p + gl) * p + i] = ok && i <= gl ? row[i] : 0.0;
    }
  if (gl == 0) {
    double rss = ydy[c];
    if (ok) {
#pragma unroll
      for (int k = 0; k < GW; ++k)
        if (k < p) rss -= b[k] * beta[k];
      if (rss < 0) rss = 0;
    }
    rss_out[g] = rss;
    delta_out[g] = st[c].d;
#pragma unroll
    for (int k = 0; k < GW; ++k)
      if (k < p) chi0_out[g * p + k] = ok ? beta[k] : 0.0;
  }
}

// Gene-side operands, one block per gene: rows (w o r~), (w o X~_k), w, each
// FP16 hi/lo with its own power-of-two scale; unscale[] = factors that turn
// the accumulators back into NUM, a_k, gg.
__global__ void lmm_gene_ops_kernel(const double* __restrict__ Ytil, const double* __restrict__ Xtil,
                                    const double* __restrict__ lam, const double* __restrict__ delta,
                                    const double* __restrict__ chi0, int n, int p, int G,
                                    const int* __restrict__ gene_row, int k_pad, float s1, float s2,
                                    __half* const* hi, __half* const* lo, float* unscale) {
  const int g = blockIdx.x;
  if (g >= G) return;
  const int64_t row = gene_row ? gene_row[g] : g;  // operand row
  const int nops = p + 2;
  __shared__ double mx[kMaxPLmm + 2][8];
  __shared__ double sc[kMaxPLmm + 2];
  const double d = delta[g];
  const double* yt = Ytil + static_cast<int64_t>(g) * n;
  double c0[kMaxPLmm];
  for (int k = 0; k < p; ++k) c0[k] = chi0[static_cast<int64_t>(g) * p + k];
  auto value = [&](int op, int i) -> double {
    if (i >= n) return 0.0;
    double v = d * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    const double w = 1.0 / v;
    if (op == 0) {
      double r = yt[i];
      for (int k = 0; k < p; ++k) r -= Xtil[static_cast<int64_t>(k) * n + i] * c0[k];
      return w * r;
    }
    if (op <= p) return w * Xtil[static_cast<int64_t>(op - 1) * n + i];
    return w;
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int op = 0; op < nops; ++op) {
    double m = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fabs(value(op, i)));
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) mx[op][warp] = m;
  }
  __syncthreads();
  if (threadIdx.x < nops) {
    double m = 0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) m = fmax(m, mx[threadIdx.x][w]);
    int e = 0;
    if (m > 0) e = 10 - static_cast<int>(floor(log2(m)));
    sc[threadIdx.x] = ldexp(1.0, e);
    const double side = threadIdx.x == nops - 1 ? s2 : s1;
    unscale[static_cast<int64_t>(g) * nops + threadIdx.x] = static_cast<float>(1.0 / (ldexp(1.0, e) * side));
  }
  __syncthreads();
  for (int op = 0; op < nops; ++op) {
    const double s = sc[op];
    for (int i = threadIdx.x; i < k_pad; i += blockDim.x) {
      const double v = value(op, i) * s;
      const __half h = __double2half(v);
      hi[op][row * k_pad + i] = h;
      lo[op][row * k_pad + i] = __double2half(v - static_cast<double>(__half2float(h)));
    }
  }
}

// Gene-side vectors of the exact-operand scan, one block per gene, in
// eigen-coordinates: column (p + 1) g of W is w o r~ and column
// (p + 1) g + 1 + k is w o X~_k, with w = 1 / max(delta lambda + 1, 1e-12);
// Q W then holds u = Q (w o r~) and v_k = Q (w o X~_k).
__global__ void lmm_uv_w_kernel(const double* __restrict__ Ytil, const double* __restrict__ Xtil,
                                const double* __restrict__ lam, const double* __restrict__ delta,
                                const double* __restrict__ chi0, int n, int p, int G, double* W) {
  const int g = blockIdx.x;
  if (g >= G) return;
  const double d = delta[g];
  const double* yt = Ytil + static_cast<int64_t>(g) * n;
  const double* c0 = chi0 + static_cast<int64_t>(g) * p;
  double* out = W + static_cast<int64_t>(g) * (p + 1) * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double v = d * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    double r = yt[i];
    for (int k = 0; k < p; ++k) {
      const double x = Xtil[static_cast<int64_t>(k) * n + i];
      r -= x * c0[k];
      out[static_cast<int64_t>(1 + k) * n + i] = x / v;
    }
    out[i] = r / v;
  }
}

// Gene-side operands of the exact-operand scan, one block per gene: rows u,
// v_0 .. v_{p-1} (columns of UV = Q W) and w, each FP16 hi/lo with its own
// power-of-two scale. unscale[] turns accumulators back into NUM, a_k (the
// SNP operand carries no scale of its own) and gg (against Gt^2 at s2).
// u and v_k are scaled to a largest entry in [8, 16), so that minus their sum
// (at most 16 n <= 32768) fits FP16 as well: it goes to column n, where the
// SNP operand holds its imputed mean, which centres each SNP inside the
// contraction.
__global__ void lmm_gene_ops_raw_kernel(const double* __restrict__ UV, const double* __restrict__ lam,
                                        const double* __restrict__ delta, int n, int p, int G,
                                        const int* __restrict__ gene_row, int k_pad, float s2, __half* const* hi,
                                        __half* const* lo, float* unscale) {
  const int g = blockIdx.x;
  if (g >= G) return;
  const int64_t row = gene_row ? gene_row[g] : g;  // operand row
  const int nops = p + 2;
  __shared__ double mx[kMaxPLmm + 2][8];
  __shared__ double sc[kMaxPLmm + 2];
  __shared__ double part[8];
  const double d = delta[g];
  const double* uv = UV + static_cast<int64_t>(g) * (p + 1) * n;
  auto value = [&](int op, int i) -> double {
    if (i >= n) return 0.0;
    if (op <= p) return uv[static_cast<int64_t>(op) * n + i];
    double v = d * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    return 1.0 / v;
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int op = 0; op < nops; ++op) {
    double m = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fabs(value(op, i)));
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) mx[op][warp] = m;
  }
  __syncthreads();
  if (threadIdx.x < nops) {
    double m = 0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) m = fmax(m, mx[threadIdx.x][w]);
    const bool centred = threadIdx.x < nops - 1;  // u and v_k
    int e = 0;
    if (m > 0) e = (centred ? 3 : 10) - static_cast<int>(floor(log2(m)));
    sc[threadIdx.x] = ldexp(1.0, e);
    const double side = centred ? 1.0 : s2;
    unscale[static_cast<int64_t>(g) * nops + threadIdx.x] = static_cast<float>(1.0 / (ldexp(1.0, e) * side));
  }
  __syncthreads();
  for (int op = 0; op < nops; ++op) {
    const double s = sc[op];
    __half* h_row = hi[op] + row * k_pad;
    __half* l_row = lo[op] + row * k_pad;
    double sum = 0.0;
    for (int i = threadIdx.x; i < k_pad; i += blockDim.x) {
      const double v = value(op, i) * s;
      const __half h = __double2half(v);
      const __half l = __double2half(v - static_cast<double>(__half2float(h)));
      h_row[i] = h;
      l_row[i] = l;
      sum += static_cast<double>(__half2float(h)) + static_cast<double>(__half2float(l));
    }
    if (op > p) break;  // w is not centred
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) part[warp] = sum;
    __syncthreads();  // every thread's writes of column n (zero) are done too
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < (blockDim.x >> 5); ++w) t += part[w];
      const __half h = __double2half(-t);
      h_row[n] = h;
      l_row[n] = __double2half(-t - static_cast<double>(__half2float(h)));
    }
    __syncthreads();
  }
}

// ------------------------------------------------------- scan epilogue
template <int P>
struct LmmEpiParams {
  int G;
  const int* order;         // GeneOrder::gene
  int64_t m;
  const float* unscale;     // [G][P+2]
  const double* ainv;       // [G][P][P]
  const double* rss_null;   // [G]
  const uint8_t* snp_ok;    // [m]
  Windows win;
  float df;
  float t_cand;
  TTable tt;
  GeneOut out;
  // NB-GLM scan only (GlmEpiParams): per kept SNP the imputation mean (the
  // SNP operand is centred), per gene sum_i r_i and the null fit's success
  const float* snp_mean;    // [m, padded to 16 + 16]
  const float* rsum;        // [G]
  const uint8_t* gene_ok;   // [G]
  // exact-operand LMM scan only (LmmRawEpiParams): per kept SNP the factor
  // alpha of the raw operand (Rotated::raw)
  const float* snp_alpha;   // [m, padded to 256 + 256]
};
// The same fields select the NB-GLM score-test epilogue (LmmEpi<P, true>).
template <int P>
struct GlmEpiParams : LmmEpiParams<P> {};
// ... and the LMM scan on the exact unrotated SNP operand (LmmEpi<P, false, true>).
template <int P>
struct LmmRawEpiParams : LmmEpiParams<P> {};
// ... and the same with gg and a_k interpolated between node deltas
// (LmmEpi<P, false, true, true>): a_k then carries no SNP factor alpha.
template <int P>
struct LmmLrEpiParams : LmmEpiParams<P> {};

// P = 1: accumulator order [NUM, gg, a_0] (the gene-side operands w o r~, w,
// w o X~_0 against Gt, Gt^2, Gt), all three read chunk by chunk. TMEM's fourth
// slot takes the next tile's NUM, whose MMAs (K = n) then run under this
// epilogue, and nothing is kept in registers from chunk to chunk. (The order
// [gg, a_0, NUM] in two phases, which P = 2 uses, kept 32 values of S per thread
// and spilled: 600 bytes of spill loads a tile.)
// P = 2: order [gg, a_0, a_1, NUM] in two phases, since four accumulators fill
// TMEM: S = gg - a' A00^-1 a of every pair of the warp's chunks first, which
// frees the gg and a slots for the next tile's MMAs, then NUM and the rest of
// the statistic.
//
// GLM = true is the NB-GLM score test on the same accumulators (unrotated
// centred dosages gc against w, w o x_k and r of the gene's null fit):
// info = S, U = NUM + mean_s * sum_i r_i, and the screened statistic is
// z^2 = U^2 / info against the normal tables.
//
// RAW = true: NUM and a_k come from the exact unrotated SNP operand
// (Rotated::raw) against the gene-side vectors u = Q (w o r~) and
// v_k = Q (w o X~_k), since Gt . (w o r~) = g . Q (w o r~); the operands
// centre each SNP themselves (padding column n), so x = alpha_s * acc.
//
// LR = true (with RAW): gg and a_k come from the node-interpolated operands
// (lmm_lr_scan), which hold each SNP's factor alpha already; NUM as RAW.
template <int P, bool GLM = false, bool RAW = false, bool LR = false>
struct LmmEpi {
  static_assert(!(GLM && RAW), "the exact-operand form is the LMM scan's");
  static_assert(!LR || RAW, "the interpolated form reads NUM from the exact operand");
  static constexpr bool kGrouped = false;
  static constexpr bool kTwoPhase = P > 1;
  static constexpr int kPhase1 = P + 1;  // gg and a_k
  static constexpr int kMaxChunks = 2;   // 16-column chunks per warp and tile
  using Params = std::conditional_t<
      GLM, GlmEpiParams<P>,
      std::conditional_t<LR, LmmLrEpiParams<P>, std::conditional_t<RAW, LmmRawEpiParams<P>, LmmEpiParams<P>>>>;
  static constexpr int kSmemBytes = kTTableSmemBytes;
  const Params& Pr;
  float* tsm;
  int gene = 0;
  int64_t snp0 = 0;
  bool gvalid = false;
  float u[P + 2];  // unscale of [NUM, a_0 .. a_{P-1}, gg] (the gene-ops order)
  float ai[P][P];
  float inv_rss = 0;
  float rs = 0;  // GLM: sum_i r_i of the gene
  // P = 2: S per pair of the warp's two chunks (0 where gg < 1e-12); two named
  // arrays picked by a select, so they stay in registers for a runtime ci
  float S0[16], S1[16];
  float u_cand;  // t_cand^2
  uint32_t tab = 0;  // screen_tables (0: none)
  GeneAcc acc;
  __device__ LmmEpi(const Params& p, const TileShape&, uint8_t* smem)
      : Pr(p), tsm(reinterpret_cast<float*>(smem)), u_cand(p.t_cand * p.t_cand) {}
  __device__ void init(int tid, int nthr) {
    if (tsm) tab = screen_tables(Pr.tt, tsm, tid, nthr);
  }
  __device__ void begin_tile(int row, int64_t s0) {
    snp0 = s0;
    gvalid = row < Pr.G;
    const int g = gene = gvalid && Pr.order ? __ldg(Pr.order + row) : row;
    if constexpr (GLM) gvalid = gvalid && Pr.gene_ok[g];  // a failed null fit tests nothing
    acc.reset();
    if (gvalid) {
      if constexpr (GLM) rs = Pr.rsum[g];
#pragma unroll
      for (int k = 0; k < P + 2; ++k) u[k] = Pr.unscale[static_cast<int64_t>(g) * (P + 2) + k];
#pragma unroll
      for (int a = 0; a < P; ++a)
#pragma unroll
        for (int b = 0; b < P; ++b) ai[a][b] = static_cast<float>(Pr.ainv[(static_cast<int64_t>(g) * P + a) * P + b]);
      if constexpr (!GLM) {
        const double r = Pr.rss_null[g];
        inv_rss = r > 0 ? static_cast<float>(1.0 / r) : 0.0f;
      }
      acc.load_window(Pr.win, g);
      acc.load_best(Pr.out, g);
    }
  }
  // Screening arithmetic in FP32 (the accumulators carry ~1e-7 relative
  // error already); printed statistics come from the FP64 refinement.
  // S of one pair from its accumulators [gg, a_0 .. a_{P-1}] (0 where gg <
  // 1e-12: p = 1, S fails the S > 1e-15 test). us: alpha of the SNP (RAW).
  template <class V>
  __device__ __forceinline__ float schur(V&& v, float us) {
    const float gg = v(0) * u[P + 1];
    float S = gg;
    float a[P];
#pragma unroll
    for (int k = 0; k < P; ++k) a[k] = v(1 + k) * (us * u[1 + k]);
#pragma unroll
    for (int x = 0; x < P; ++x)
#pragma unroll
      for (int y = 0; y < P; ++y) S = fmaf(-a[x] * ai[x][y], a[y], S);
    return gg < 1e-12f ? 0.0f : S;
  }
  // The screen of 16 pairs from NUM's accumulators and S.
  __device__ __forceinline__ void screen(int64_t s0, const float (&num_acc)[16], const float (&S)[16]) {
    const float4* al4 = reinterpret_cast<const float4*>(Pr.snp_alpha + s0);  // RAW (padded past the last tile)
    uint32_t okw[4];
    load_flags16(Pr.snp_ok + s0, okw);
    float s_min = INFINITY;
#pragma unroll
    for (int j = 0; j < 16; j += 2) s_min = min3(s_min, S[j], S[j + 1]);
    auto num_of = [&](int j) {
      float num = num_acc[j] * u[0];
      if constexpr (RAW) {
        const float4 a = __ldg(al4 + (j >> 2));
        num *= (j & 3) == 0 ? a.x : (j & 3) == 1 ? a.y : (j & 3) == 2 ? a.z : a.w;
      }
      return num;
    };
    screen_chunk(
        Pr.tt, tab, u_cand, Pr.win, Pr.out, gene, s0, all_flags16(okw) && s_min > 1e-15f,
        [&](int j) {
          const float num = num_of(j);
          if constexpr (GLM) {
            const float U = fmaf(__ldg(Pr.snp_mean + s0 + j), rs, num);
            return U * U * rcp_ftz(S[j]);  // z^2
          } else {
            const float r = num * (num * rcp_ftz(S[j])) * inv_rss;
            return Pr.df * (r * rcp_ftz(1.0f - r));  // t^2
          }
        },
        [&](int j, bool& tested) {
          tested = flag16(okw, j);  // zero past the last kept SNP
          const float num = num_of(j);
          float t2;
          if constexpr (GLM) {
            const float U = fmaf(__ldg(Pr.snp_mean + s0 + j), rs, num);
            t2 = S[j] > 1e-15f ? __fdividef(U * U, S[j]) : 0.0f;
            if (!(t2 == t2)) t2 = 0.0f;
          } else {
            const float r = num * __fdividef(num, S[j]) * inv_rss;
            const float omr = 1.0f - r;
            t2 = S[j] > 1e-15f && omr > 0.0f ? Pr.df * __fdividef(r, omr) : 0.0f;
          }
          return t2;
        },
        acc);
  }
  // P = 2, phase 1: v = [gg, a_0, a_1] of 16 pairs.
  template <int N>
  __device__ void pre_chunk(int ci, int c, const float (&v)[N][16]) {
    static_assert(N == P + 1, "phase-1 accumulators");
    float al[16];  // RAW: alpha of each SNP (the array is padded past the last tile)
    if constexpr (RAW && !LR) load16(Pr.snp_alpha + snp0 + c, al);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float us = 1.0f;
      if constexpr (RAW && !LR) us = al[j];
      const float Sj = schur([&](int k) { return v[k][j]; }, us);
      if (ci == 0) S0[j] = Sj;
      else S1[j] = Sj;
    }
  }
  // Phase 2: v = [NUM] of the same 16 pairs.
  template <int N>
  __device__ void post_chunk(int ci, int c, const float (&v)[N][16]) {
    static_assert(N == 1, "phase-2 accumulators");
    const int64_t s0 = snp0 + c;
    if (!gvalid || s0 >= Pr.m) return;
    float S[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) S[j] = ci == 0 ? S0[j] : S1[j];
    screen(s0, v[0], S);
  }
  // All accumulators of 16 pairs at once: P = 1 in its order [NUM, gg, a_0].
  template <int NACC>
  __device__ void chunk(int c, const float (&v)[NACC][16]) {
    static_assert(NACC == P + 2, "accumulators");
    all_at_once<0, 1>(c, v);
  }
  template <int NUM, int GG, int NACC>
  __device__ __forceinline__ void all_at_once(int c, const float (&v)[NACC][16]) {
    const int64_t s0 = snp0 + c;
    if (!gvalid || s0 >= Pr.m) return;
    float S[16];
    {
      float al[16];
      if constexpr (RAW && !LR) load16(Pr.snp_alpha + s0, al);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float us = 1.0f;
        if constexpr (RAW && !LR) us = al[j];
        S[j] = schur([&](int k) { return v[GG + k][j]; }, us);
      }
    }
    screen(s0, v[NUM], S);
  }
  __device__ void end_tile() {
    if (gvalid) acc.flush(Pr.out, gene);
  }
  __device__ void finish() {}
};

// The CUDA-core comparator hands over its accumulators as [gg, a_0 .., NUM].
template <int P>
struct LmmSimtEpi : LmmEpi<P> {
  using LmmEpi<P>::LmmEpi;
  template <int NACC>
  __device__ void chunk(int c, const float (&v)[NACC][16]) {
    this->template all_at_once<P + 1, 0>(c, v);
  }
};

// ------------------------------------- node-interpolated gg and a_k (p <= 2)
// The weights w_i = 1 / (1 + delta lambda_i) of a gene enter gg and a_k only
// through delta, and as functions of a = ln(delta) they are analytic in a
// strip of half-width pi around the real axis. So on an interval of a of
// length <= 3, the Lagrange interpolant through 12 Chebyshev-Lobatto nodes
// reproduces every w_i to 1.1e-7 relative at worst (where delta lambda_i is
// near 8), below the 2^-22 to which the FP16 hi/lo pair holds w itself, and
// far closer on shorter intervals; with it
//     gg(s, g) = sum_j l_j(a_g) gg(s, node j),   a_k likewise,
// where gg(s, node j) is the contraction for a "node gene" of delta_j. The
// node pass computes those for the <= 128 nodes that cover the scan's genes
// (one gene-side tile), and the scan then forms gg and a_k with K = the node
// count instead of n. The Lebesgue constants keep |l_j| sums below ~5, so the
// interpolation adds at most a few FP32 roundings.

// Node pass epilogue: rows = nodes, accumulators [gg, a_0 .. a_{P-1}] of
// every kept SNP in FP32 (gg as the scan forms it, a_k with the SNP's alpha)
// into val[s][kind * kn + node] (kind 0 = gg, 1 + k = a_k), and per column
// the largest magnitude (colmax, FP32 bits; non-negative floats order as
// unsigned integers).
template <int P>
struct LmmNodeEpiParams {
  int n_nodes;
  int64_t m;
  int kn, kb;               // node columns per kind (64 or 128); kb = (P + 1) kn
  const float* unscale;     // [nodes][P + 2] in the gene-ops order [NUM, a_0 .., gg]
  const float* snp_alpha;   // [m, padded to 256 + 256]
  float* val;               // [m][kb]
  unsigned int* colmax;     // [kb]
};

template <int P>
struct LmmNodeEpi {
  static constexpr bool kGrouped = false;
  static constexpr int kSmemBytes = 0;
  using Params = LmmNodeEpiParams<P>;
  const Params& Pr;
  int node = 0;
  int64_t snp0 = 0;
  bool valid = false;
  float u[P + 1];   // unscale of [gg, a_0 ..]
  float mx[P + 1];  // largest magnitude of each kind over the tile
  __device__ LmmNodeEpi(const Params& p, const TileShape&, uint8_t*) : Pr(p) {}
  __device__ void init(int, int) {}
  __device__ void begin_tile(int g, int64_t s0) {
    node = g;
    snp0 = s0;
    valid = g < Pr.n_nodes;
#pragma unroll
    for (int k = 0; k <= P; ++k) mx[k] = 0.0f;
    if (valid) {
      u[0] = Pr.unscale[static_cast<int64_t>(g) * (P + 2) + P + 1];
#pragma unroll
      for (int k = 0; k < P; ++k) u[1 + k] = Pr.unscale[static_cast<int64_t>(g) * (P + 2) + 1 + k];
    }
  }
  template <int N>
  __device__ void chunk(int c, const float (&v)[N][16]) {
    static_assert(N == P + 1, "node pass accumulators");
    const int64_t s0 = snp0 + c;
    if (!valid || s0 >= Pr.m) return;
    float al[16];
    load16(Pr.snp_alpha + s0, al);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int64_t s = s0 + j;
      if (s < Pr.m) {
        float* row = Pr.val + s * Pr.kb + node;
        const float gg = v[0][j] * u[0];
        row[0] = gg;
        mx[0] = fmaxf(mx[0], fabsf(gg));
#pragma unroll
        for (int k = 0; k < P; ++k) {
          const float a = v[1 + k][j] * (u[1 + k] * al[j]);
          row[static_cast<int64_t>(1 + k) * Pr.kn] = a;
          mx[1 + k] = fmaxf(mx[1 + k], fabsf(a));
        }
      }
    }
  }
  __device__ void end_tile() {
    if (!valid) return;
#pragma unroll
    for (int k = 0; k <= P; ++k)
      if (mx[k] > 0.0f) atomicMax(Pr.colmax + k * Pr.kn + node, __float_as_uint(mx[k]));
  }
  __device__ void finish() {}
};

// Scale of each node column: a power of two that takes its largest value
// into [2^14, 2^15) (0 for a column that is zero throughout, and for the
// padding columns).
__global__ void lr_sigma_kernel(const unsigned int* __restrict__ colmax, int kb, float* sigma) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kb) return;
  const float mx = __uint_as_float(colmax[i]);
  sigma[i] = mx > 0.0f ? ldexpf(1.0f, min(14 - ilogbf(mx), 100)) : 0.0f;
}

// The SNP-side operand of the interpolated accumulators: val * sigma of its
// column as FP16 hi + lo, four values per thread (kb is a multiple of 64).
// Columns of scale 0 are written as 0 without reading val (padding columns
// are never written by the node pass).
__global__ void lr_split_kernel(const float* __restrict__ val, int64_t total, int kb,
                                const float* __restrict__ sigma, __half* hi, __half* lo) {
  const int64_t n4 = total / 4;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c0 = static_cast<int>((4 * i) % kb);
    float x[4];
    const float4 sg = *reinterpret_cast<const float4*>(sigma + c0);
    const float sv[4] = {sg.x, sg.y, sg.z, sg.w};
    const bool any = sv[0] != 0.0f || sv[1] != 0.0f || sv[2] != 0.0f || sv[3] != 0.0f;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (any) v = reinterpret_cast<const float4*>(val)[i];
    const float vv[4] = {v.x, v.y, v.z, v.w};
    uint32_t hw[2], lw[2];
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = sv[t] != 0.0f ? vv[t] * sv[t] : 0.0f;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const __half h0 = __float2half_rn(x[2 * t]), h1 = __float2half_rn(x[2 * t + 1]);
      const __half l0 = __float2half_rn(x[2 * t] - __half2float(h0));
      const __half l1 = __float2half_rn(x[2 * t + 1] - __half2float(h1));
      hw[t] = static_cast<uint32_t>(__half_as_ushort(h0)) | (static_cast<uint32_t>(__half_as_ushort(h1)) << 16);
      lw[t] = static_cast<uint32_t>(__half_as_ushort(l0)) | (static_cast<uint32_t>(__half_as_ushort(l1)) << 16);
    }
    reinterpret_cast<uint2*>(hi)[i] = make_uint2(hw[0], hw[1]);
    reinterpret_cast<uint2*>(lo)[i] = make_uint2(lw[0], lw[1]);
  }
}

constexpr int kLrNodes = 12;     // Chebyshev-Lobatto nodes per interval of ln(delta)
constexpr double kLrSpan = 3.0;  // longest interval of ln(delta)

// Gene-side operands of the interpolated accumulators, one thread per gene:
// the Lagrange weights l_j(a) of the gene's interval (a = ln delta, nodes
// node_a[base .. base + kLrNodes), base = q (kLrNodes - 1)) over each kind's
// column scale, times a power of two per gene and kind, as FP16 hi + lo at
// [g][kind * kn + base + j] (rows zeroed beforehand), and that power's
// inverse as the unscale of gg (kind 0) and a_k (kind 1 + k).
__global__ void lr_coef_kernel(const double* __restrict__ delta, int G, const double* __restrict__ node_a,
                               double a0, double h, int nint, const float* __restrict__ sigma, int kn, int kb,
                               int P, const int* __restrict__ gene_row, __half* hi, __half* lo, float* unscale) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G) return;
  double a = log(fmax(delta[g], 1e-300));
  if (!(a == a)) a = a0;
  int q = static_cast<int>(floor((a - a0) / h));
  q = q < 0 ? 0 : (q >= nint ? nint - 1 : q);
  const int base = q * (kLrNodes - 1);
  double l[kLrNodes];
#pragma unroll
  for (int j = 0; j < kLrNodes; ++j) {
    double t = 1.0;
#pragma unroll
    for (int i = 0; i < kLrNodes; ++i)
      if (i != j) t *= (a - node_a[base + i]) / (node_a[base + j] - node_a[base + i]);
    l[j] = t;
  }
  for (int kind = 0; kind <= P; ++kind) {
    const float* sg = sigma + kind * kn + base;
    double mx = 0.0;
#pragma unroll
    for (int j = 0; j < kLrNodes; ++j)
      if (sg[j] != 0.0f) mx = fmax(mx, fabs(l[j] / static_cast<double>(sg[j])));
    const double sc = mx > 0.0 ? ldexp(1.0, 10 - ilogb(mx)) : 1.0;
    const int64_t row = gene_row ? gene_row[g] : g;
    __half* hr = hi + row * kb + kind * kn + base;
    __half* lr = lo + row * kb + kind * kn + base;
#pragma unroll
    for (int j = 0; j < kLrNodes; ++j) {
      const double y = sg[j] != 0.0f ? l[j] / static_cast<double>(sg[j]) * sc : 0.0;
      const __half hv = __double2half(y);
      hr[j] = hv;
      lr[j] = __double2half(y - static_cast<double>(__half2float(hv)));
    }
    unscale[static_cast<int64_t>(g) * (P + 2) + (kind == 0 ? P + 1 : kind)] = static_cast<float>(1.0 / sc);
  }
}

// ---------------------------------------- any number of covariates (p >= 3)
// With A00 = X~'W X~ and U U' = A00^-1 (Cholesky of the REML kernel's ainv),
// a' A00^-1 a = |U' a|^2 and U' a = Gt'(w o X~U): each covariate column
// becomes one plain accumulator a~_k = Gt'(w o (X~U)_k), and
//     S = gg - sum_k a~_k^2.
// The p + 2 accumulators exceed what TMEM holds for one tile, so the tile kernel
// runs them in groups of two, in the order [gg, a~_0 .. a~_{p-1}, NUM]: this
// epilogue keeps only the running S of its pairs across the groups, and NUM ends
// the tile. Tiles are 128 SNPs wide: per K chunk of an accumulator (12 MMAs) an SM
// then moves 160 KB through shared memory for 128 x 128 pairs, or 120 KB on SM
// pairs, where the 64-wide tiles that NUM and S of a thread once limited it to
// moved 120 KB for half as many; shared memory's 128 bytes a cycle is what bounds
// the kernel. NB-GLM scan (n = 1000, p = 3, 2e8 tests) 6.3 -> 4.3 ms (1.42 PFLOP/s
// issued), LMM scan (n = 1000, p = 6, 2e8 tests) 10.0 -> 6.8 ms (1.44 PFLOP/s).
//
// Both passes (largest entry of each operand, then its halves) form a sample's
// values from its weight and covariates in registers: one division and p PM fused
// multiply-adds (those above U's diagonal add exact zeros: a loop over whole
// columns keeps x in registers), U broadcast from shared memory as pairs, two
// samples a thread. A pass that takes an operand at a time divides and reads the
// covariates p + 2 times for the same. PM: p rounded up.
// n = 1000, p = 16, 8,000 genes: 2.48 -> 0.97 ms (one thread used to factorise).
template <int PM>
__global__ void __launch_bounds__(256) lmm_gene_ops_orth_kernel(
    const double* __restrict__ Ytil, const double* __restrict__ Xtil, const double* __restrict__ lam,
    const double* __restrict__ delta, const double* __restrict__ chi0, const double* __restrict__ ainv, int n, int p,
    int G, const int* __restrict__ gene_row, int k_pad, float s1, float s2, __half* const* hi, __half* const* lo,
    float* unscale) {
  constexpr int NS = PM <= 16 ? 2 : 1;  // samples per thread and step
  const int g = blockIdx.x;
  if (g >= G) return;
  const int64_t row = gene_row ? gene_row[g] : g;  // operand row
  const int nops = p + 2;
  __shared__ double mx[PM + 2][8];
  __shared__ double sc[PM + 2];
  __shared__ double c0[PM];
  __shared__ __align__(16) double Ut[PM][PM];  // transpose of the lower Cholesky factor of ainv[g]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t = threadIdx.x; t < PM * PM; t += blockDim.x) Ut[t / PM][t % PM] = 0.0;
  for (int k = threadIdx.x; k < PM; k += blockDim.x) c0[k] = k < p ? chi0[static_cast<int64_t>(g) * p + k] : 0.0;
  for (int t = threadIdx.x; t < (PM + 2) * 8; t += blockDim.x) mx[t / 8][t % 8] = 0.0;
  __syncthreads();
  if (warp == 0) {  // lane i has row i
    const double* A = ainv + static_cast<int64_t>(g) * p * p;
    for (int j = 0; j < p; ++j) {
      double v = 0.0;
      if (lane >= j && lane < p) {
        v = A[lane * p + j];
        for (int k = 0; k < j; ++k) v -= Ut[k][lane] * Ut[k][j];
      }
      double d = __shfl_sync(0xffffffffu, v, j);
      d = d > 0 ? sqrt(d) : 0.0;  // A00 is positive definite wherever REML succeeded
      if (lane >= j && lane < p) Ut[j][lane] = lane == j ? d : (d > 0 ? v / d : 0.0);
      __syncwarp();
    }
  }
  __syncthreads();
  const double d = delta[g];
  const double* yt = Ytil + static_cast<int64_t>(g) * n;
  // out(op, values) of samples i0 .. i0 + NS - 1, zero past n
  auto values = [&](int i0, auto&& out) {
    double w[NS], r[NS], x[NS][PM];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const int i = i0 + s;
      const bool in = i < n;
      double v = in ? d * lam[i] + 1.0 : 1.0;
      if (v < 1e-12) v = 1e-12;
      w[s] = in ? 1.0 / v : 0.0;
      r[s] = in ? yt[i] : 0.0;
#pragma unroll
      for (int k = 0; k < PM; ++k) x[s][k] = in && k < p ? Xtil[static_cast<int64_t>(k) * n + i] : 0.0;
#pragma unroll
      for (int k = 0; k < PM; ++k) r[s] -= x[s][k] * c0[k];
      r[s] = w[s] * r[s];
    }
    out(0, r);
    out(1, w);
#pragma unroll 1
    for (int k = 0; k < p; ++k) {
#pragma unroll
      for (int s = 0; s < NS; ++s) r[s] = 0.0;
#pragma unroll
      for (int l = 0; l < PM; ++l) {
        const double u = Ut[k][l];
#pragma unroll
        for (int s = 0; s < NS; ++s) r[s] += x[s][l] * u;
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) r[s] = w[s] * r[s];
      out(2 + k, r);
    }
  };
  for (int base = 0; base < n; base += NS * blockDim.x)  // the same steps in every lane
    values(base + NS * threadIdx.x, [&](int op, const double (&v)[NS]) {
      double m = 0.0;
#pragma unroll
      for (int s = 0; s < NS; ++s) m = fmax(m, fabs(v[s]));
      // the warp's largest: non-negative doubles are ordered as their words
      const unsigned hw = static_cast<unsigned>(__double2hiint(m));
      const unsigned mh = __reduce_max_sync(0xffffffffu, hw);
      const unsigned ml =
          __reduce_max_sync(0xffffffffu, hw == mh ? static_cast<unsigned>(__double2loint(m)) : 0u);
      if (lane == 0) mx[op][warp] = fmax(mx[op][warp], __hiloint2double(static_cast<int>(mh), static_cast<int>(ml)));
    });
  __syncthreads();
  if (threadIdx.x < nops) {
    double m = 0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) m = fmax(m, mx[threadIdx.x][w]);
    int e = 0;
    if (m > 0) e = 10 - static_cast<int>(floor(log2(m)));
    sc[threadIdx.x] = ldexp(1.0, e);
    const double side = threadIdx.x == 1 ? s2 : s1;  // gg pairs with Gt^2, the rest with Gt
    unscale[static_cast<int64_t>(g) * nops + threadIdx.x] = static_cast<float>(1.0 / (ldexp(1.0, e) * side));
  }
  __syncthreads();
  for (int i = NS * threadIdx.x; i < k_pad; i += NS * blockDim.x)
    values(i, [&](int op, const double (&v)[NS]) {
      const double s = sc[op];
      __half h[NS], l[NS];
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const double a = v[j] * s;
        h[j] = __double2half(a);
        l[j] = __double2half(a - static_cast<double>(__half2float(h[j])));
      }
      if constexpr (NS == 2) {
        *reinterpret_cast<__half2*>(hi[op] + row * k_pad + i) = __halves2half2(h[0], h[1]);
        *reinterpret_cast<__half2*>(lo[op] + row * k_pad + i) = __halves2half2(l[0], l[1]);
      } else {
        hi[op][row * k_pad + i] = h[0];
        lo[op][row * k_pad + i] = l[0];
      }
    });
}

struct LmmGroupEpiParams {
  int G;
  const int* order;         // GeneOrder::gene
  int64_t m;
  int n_acc;                // p + 2
  const float* unscale;     // [G][n_acc]: NUM, gg, a~_0 .. a~_{p-1} (the gene-ops order)
  const double* rss_null;   // [G]
  const uint8_t* snp_ok;    // [m]
  Windows win;
  float df;
  float t_cand;
  TTable tt;
  GeneOut out;
  const float* snp_mean;    // GLM only, as in LmmEpiParams
  const float* rsum;
  const uint8_t* gene_ok;
};
struct GlmGroupEpiParams : LmmGroupEpiParams {};

// GLM = true: the NB-GLM score test, as in LmmEpi.
template <bool GLM>
struct LmmGroupEpiT {
  static constexpr bool kGrouped = true;
  static constexpr int kTileN = 128;
  static constexpr int kGroup = 2;      // accumulators per group: two groups in TMEM
  static constexpr int kMaxChunks = 2;  // 16-column chunks per warp and tile
  using Params = std::conditional_t<GLM, GlmGroupEpiParams, LmmGroupEpiParams>;
  static constexpr int kSmemBytes = kTTableSmemBytes;
  const Params& Pr;
  float* tsm;
  int gene = 0;
  int64_t snp0 = 0;
  bool gvalid = false;
  float inv_rss = 0;
  float rs = 0;  // GLM: sum_i r_i of the gene
  // running S per pair of the warp's two chunks; two named arrays picked by a
  // select, so they stay in registers for a runtime ci
  float S0[16], S1[16];
  float u_cand;  // t_cand^2
  uint32_t tab = 0;  // screen_tables (0: none)
  GeneAcc acc;
  __device__ LmmGroupEpiT(const Params& p, const TileShape&, uint8_t* smem)
      : Pr(p), tsm(reinterpret_cast<float*>(smem)), u_cand(p.t_cand * p.t_cand) {}
  __device__ void init(int tid, int nthr) {
    tab = screen_tables(Pr.tt, tsm, tid, nthr);
  }
  __device__ void begin_tile(int row, int64_t s0) {
    snp0 = s0;
    gvalid = row < Pr.G;
    const int g = gene = gvalid && Pr.order ? __ldg(Pr.order + row) : row;
    if constexpr (GLM) gvalid = gvalid && Pr.gene_ok[g];
    acc.reset();
    if (gvalid) {
      if constexpr (GLM) {
        rs = Pr.rsum[g];
      } else {
        const double r = Pr.rss_null[g];
        inv_rss = r > 0 ? static_cast<float>(1.0 / r) : 0.0f;
      }
      acc.load_window(Pr.win, g);
      acc.load_best(Pr.out, g);
    }
  }
  // accumulator j of this tile for the 16 columns at c
  __device__ void acc_chunk(int j, int ci, int c, const float (&v)[16]) {
    if (!gvalid) return;
    const float* us = Pr.unscale + static_cast<int64_t>(gene) * Pr.n_acc;
    if (j == Pr.n_acc - 1) {
      screen(ci, snp0 + c, v, __ldg(us));
      return;
    }
    const float f = __ldg(us + j + 1);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float x = v[i] * f;
      float s;
      if (j == 0) s = x < 1e-12f ? -INFINITY : x;  // gg < 1e-12: p = 1
      else s = fmaf(-x, x, ci == 0 ? S0[i] : S1[i]);
      if (ci == 0) S0[i] = s;
      else S1[i] = s;
    }
  }
  // NUM of the 16 pairs, the last accumulator: their t, tail and per-gene updates
  __device__ __forceinline__ void screen(int ci, int64_t s0, const float (&v)[16], float us) {
    if (s0 >= Pr.m) return;
    uint32_t okw[4];
    load_flags16(Pr.snp_ok + s0, okw);
    float S[16], s_min = INFINITY;
#pragma unroll
    for (int j = 0; j < 16; ++j) S[j] = ci == 0 ? S0[j] : S1[j];
#pragma unroll
    for (int j = 0; j < 16; j += 2) s_min = min3(s_min, S[j], S[j + 1]);
    screen_chunk(
        Pr.tt, tab, u_cand, Pr.win, Pr.out, gene, s0, all_flags16(okw) && s_min > 1e-15f,
        [&](int j) {
          const float num = v[j] * us;
          if constexpr (GLM) {
            const float U = fmaf(__ldg(Pr.snp_mean + s0 + j), rs, num);
            return U * U * rcp_ftz(S[j]);  // z^2
          } else {
            const float r = num * (num * rcp_ftz(S[j])) * inv_rss;
            return Pr.df * (r * rcp_ftz(1.0f - r));  // t^2
          }
        },
        [&](int j, bool& tested) {
          tested = flag16(okw, j);  // zero past the last kept SNP
          const float num = v[j] * us;
          float t2;
          if constexpr (GLM) {
            const float U = fmaf(__ldg(Pr.snp_mean + s0 + j), rs, num);
            t2 = S[j] > 1e-15f ? __fdividef(U * U, S[j]) : 0.0f;
            if (!(t2 == t2)) t2 = 0.0f;
          } else {
            const float r = num * __fdividef(num, S[j]) * inv_rss;
            const float omr = 1.0f - r;
            t2 = S[j] > 1e-15f && omr > 0.0f ? Pr.df * __fdividef(r, omr) : 0.0f;
          }
          return t2;
        },
        acc);
  }
  __device__ void end_tile() {
    if (gvalid) acc.flush(Pr.out, gene);
  }
  __device__ void finish() {}
};

using LmmGroupEpi = LmmGroupEpiT<false>;
using GlmGroupEpi = LmmGroupEpiT<true>;

// subset gate for the LMM scan (src/scan_common.cpp:133-151)
__global__ void snp_gate_kernel(const int64_t* __restrict__ kept, int64_t m, int n, const double* __restrict__ mu,
                                const int32_t* __restrict__ n_miss, const double* __restrict__ s1,
                                const double* __restrict__ s2, uint8_t* ok) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= m) return;
  const int64_t s = kept[r];
  const double mus = mu[s];
  const int k = n_miss[s];
  const double sum = s1[s] + k * mus;
  const double sum2 = s2[s] + k * mus * mus;
  double af = (sum / n) / 2.0;
  af = fmin(fmax(af, 0.0), 1.0);
  const double maf = af > 0.5 ? 1.0 - af : af;
  const double var = sum2 / n - (sum / n) * (sum / n);
  ok[r] = (maf < 1e-12 || var < 1e-12) ? 0 : 1;
}

// raw dosages of listed kept SNPs, column-major [n, u]
__global__ void listed_pairs_kernel(const int2* __restrict__ pairs, const int* __restrict__ list, int n,
                                    int2* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = pairs[list[i]];
}
__global__ void raw_dosage_kernel(GenoRows src, const int32_t* __restrict__ col, int n,
                                  const int64_t* __restrict__ kept, const double* __restrict__ mu,
                                  const int* __restrict__ snps, int u, double* out) {
  const int64_t tot = static_cast<int64_t>(u) * n;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < tot;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(e / n);
    const int i = static_cast<int>(e - static_cast<int64_t>(c) * n);
    const int64_t s = kept[snps[c]];
    const double d = src.dosage(s, col[i]);
    out[e] = isnan(d) ? mu[s] : d;
  }
}

// ------------------------------------- exact Q'g on the tensor cores
// Gt = Q'g of the listed SNPs in FP64, for 2-bit rows: the dosages are 0, 1 or
// 2, so with each eigenvector cut into digits of 12 bits
//     q_i 2^s = d_1 + d_2 / 4096 + ... + d_5 / 4096^4,   d_k integers, |d_k| <= 2048
// every sum over i of d_k g_i is an integer of at most 4096 n < 2^24 (n <=
// kQgMaxN) and therefore exact in the tensor cores' FP32 accumulators. The five
// sums of an eigenvector meet in FP64. The digits cover 2^-60 of the
// eigenvector's largest entry, so the result is at least as close to the exact
// sum as a DGEMM's, whose products and partial sums round. Missing calls are 0
// in g; a second pass contracts the 0 / 1 mask of missing calls and adds mu
// times its sums. The DGEMM this replaces was half of the refinement: n = 2000,
// 52,000 SNPs 11.4 -> 4 ms.
// Digit rows: eigenvector j has rows 16 (j / 3) + 5 (j % 3) + k, so 16 rows hold
// three whole eigenvectors (and one zero row).
constexpr int kQgDigits = 5;
constexpr int kQgMaxN = 4095;
// From this n^2 u on (a DGEMM of 0.6 ms): below, the digits, the passes' launches
// and their status checks cost what they save (n = 1,201, 2,400 SNPs: refinement
// 0.74 ms with the DGEMM, 0.76 without).
constexpr int64_t kQgMinWork = int64_t(10) << 30;
constexpr int kQgDgemmCols = 2048;
__host__ __device__ constexpr int64_t qg_rows(int n) { return static_cast<int64_t>((n + 2) / 3) * 16; }

__global__ void __launch_bounds__(256)
    q_digits_kernel(const double* __restrict__ Q, int n, int k_pad, __half* out, double* scale) {
  __shared__ double red[8];
  const int j = blockIdx.x;
  const double* q = Q + static_cast<int64_t>(j) * n;
  double mx = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) mx = fmax(mx, fabs(q[i]));
  for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = red[0];
  for (int w = 1; w < 8; ++w) mx = fmax(mx, red[w]);
  const int e = mx > 0 ? 10 - ilogb(mx) : 0;  // the largest entry times 2^e lies in [1024, 2048)
  if (threadIdx.x == 0) scale[j] = ldexp(1.0, -e);
  __half* rows = out + (static_cast<int64_t>(j / 3) * 16 + (j % 3) * kQgDigits) * k_pad;
  for (int i = threadIdx.x; i < k_pad; i += 256) {
    double x = i < n ? ldexp(q[i], e) : 0.0;
#pragma unroll
    for (int k = 0; k < kQgDigits; ++k) {
      const double d = rint(x);
      rows[static_cast<int64_t>(k) * k_pad + i] = __double2half(d);
      x = (x - d) * 4096.0;  // exact
    }
  }
}

// Dosages of the listed kept SNPs as FP16 rows (missing calls 0) and the mask
// of missing calls (mask null: not wanted), one warp per SNP.
__global__ void __launch_bounds__(256)
    listed_dosage_kernel(GenoRows src, const int32_t* __restrict__ col, int n, int k_pad,
                         const int64_t* __restrict__ kept, const int* __restrict__ snps, int u, __half* dose,
                         __half* mask) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= u) return;
  const int64_t s = kept[snps[c]];
  for (int k0 = lane * 8; k0 < k_pad; k0 += 256) {
    uint32_t dw[4] = {0, 0, 0, 0}, mw[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = k0 + j;
      const double d = k < n ? src.dosage(s, __ldg(col + k)) : 0.0;
      if (isnan(d)) mw[j / 2] |= 0x3C00u << (16 * (j & 1));  // 1.0
      else dw[j / 2] |= static_cast<uint32_t>(__half_as_ushort(__double2half(d))) << (16 * (j & 1));
    }
    const int64_t o = static_cast<int64_t>(c) * k_pad + k0;
    *reinterpret_cast<uint4*>(dose + o) = make_uint4(dw[0], dw[1], dw[2], dw[3]);
    if (mask) *reinterpret_cast<uint4*>(mask + o) = make_uint4(mw[0], mw[1], mw[2], mw[3]);
  }
}

// Rows = digit rows, columns = listed SNPs; out[c * n + j] = the five digit sums
// of eigenvector j, or += mu_c times them (the mask's pass). The digits of an eigenvector lie in five neighbouring lanes,
// so a warp passes its 32 x 16 accumulators through shared memory and each lane
// forms three outputs, consecutive lanes those of consecutive eigenvectors: no
// conversion to FP64 (8 issue cycles a warp) is done twice, and a column is
// stored as 48 contiguous bytes.
struct QgEpiParams {
  int n, u;
  const double* scale;  // [n]
  const double* mu;     // [m_all] imputation means (null: the dosages' pass)
  const int64_t* kept;
  const int* snps;
  double* out;
};

struct QgEpi {
  static constexpr bool kGrouped = false;
  static constexpr int kWarpFloats = 32 * 16;  // row r, column i at 16 r + (i ^ (r % 16))
  static constexpr int kSmemBytes = kEpiWarps * kWarpFloats * 4;
  using Params = QgEpiParams;
  const Params& P;
  float* buf;
  int64_t c0 = 0;
  int j0 = 0;  // the warp's first eigenvector
  __device__ QgEpi(const Params& p, const TileShape&, uint8_t* smem)
      : P(p), buf(reinterpret_cast<float*>(smem) + ((threadIdx.x >> 5) - 2) * kWarpFloats) {}
  __device__ void init(int, int) {}
  __device__ void begin_tile(int row, int64_t col) {
    c0 = col;
    j0 = 3 * (row / 32) * 2;
  }
  template <int NACC>
  __device__ void chunk(int cc, const float (&v)[NACC][16]) {
    const int lane = threadIdx.x & 31;
    __syncwarp();  // the previous chunk has been read
#pragma unroll
    for (int i = 0; i < 16; ++i) buf[lane * 16 + (i ^ (lane & 15))] = v[0][i];
    __syncwarp();
    double* dst[3];
    double x[3], mu[3], before[3];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const int o = lane + 32 * t, i = o / 6, e = o % 6;  // column i, eigenvector j0 + e
      const int64_t c = c0 + cc + i;
      dst[t] = c < P.u && j0 + e < P.n ? P.out + c * P.n + j0 + e : nullptr;
      if (P.mu && dst[t]) {
        mu[t] = P.mu[P.kept[P.snps[c]]];
        before[t] = *dst[t];
      }
      const float* b = buf + 256 * (e / 3);
      const int r0 = kQgDigits * (e % 3);
      auto digit = [&](int k) { return static_cast<double>(b[(r0 + k) * 16 + (i ^ (r0 + k))]); };
      x[t] = digit(kQgDigits - 1);
#pragma unroll
      for (int k = kQgDigits - 2; k >= 0; --k) x[t] = fma(x[t], 1.0 / 4096.0, digit(k));
      if (dst[t]) x[t] *= P.scale[j0 + e];
    }
#pragma unroll
    for (int t = 0; t < 3; ++t)
      if (dst[t]) *dst[t] = P.mu ? fma(mu[t], x[t], before[t]) : x[t];
  }
  __device__ void end_tile() {}
  __device__ void finish() {}
};

// The pairs [first, end) of a list, whose sums stand at the front of a buffer.
struct PairRange {
  int first, end;
};

// One warp per (gene, snp) pair from the FP64 rotated raw dosage Gt = Q'g:
// gg = Gt'W Gt, yg = Gt'W y~, a = X~'W Gt with W = diag(1 / (delta lambda + 1)),
// then the pair's printed statistics (test_lmm_gtil, src/scan_trans_lmm.cpp:11-40).
// FP64 sums [gg, yg, a_0 .. a_{p-1}] of listed (gene, snp) pairs, one warp per pair
// (p <= PM, the a_k in registers: an array indexed by a runtime p lives in local
// memory and chains every sample's update through it).
template <int PM>
__global__ void lmm_pair_sums_kernel(const double* __restrict__ Gt, int n, const int* __restrict__ pair_col,
                                     const int2* __restrict__ pairs, PairRange pr, const double* __restrict__ Ytil,
                                     const double* __restrict__ Xtil, int p, const double* __restrict__ lam,
                                     const double* __restrict__ delta, double* __restrict__ sums) {
  const int lane = threadIdx.x & 31;
  const int w = pr.first + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= pr.end) return;
  const int g = pairs[w].x;
  const double* gt = Gt + static_cast<int64_t>(pair_col[w]) * n;
  const double* yt = Ytil + static_cast<int64_t>(g) * n;
  const double d = delta[g];
  double gg = 0, yg = 0, a[PM];
#pragma unroll
  for (int k = 0; k < PM; ++k) a[k] = 0;
#pragma unroll(PM <= 4 ? 8 : 2)
  for (int i = lane; i < n; i += 32) {
    double v = d * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    const double dg = gt[i] / v;
    gg += dg * gt[i];
    yg += dg * yt[i];
#pragma unroll
    for (int k = 0; k < PM; ++k)
      if (k < p) a[k] += Xtil[static_cast<int64_t>(k) * n + i] * dg;
  }
  for (int o = 16; o; o >>= 1) {
    gg += __shfl_xor_sync(0xffffffffu, gg, o);
    yg += __shfl_xor_sync(0xffffffffu, yg, o);
#pragma unroll
    for (int k = 0; k < PM; ++k)
      if (k < p) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
  }
  if (lane != 0) return;
  double* out = sums + static_cast<int64_t>(w - pr.first) * (p + 2);
  out[0] = gg;
  out[1] = yg;
#pragma unroll
  for (int k = 0; k < PM; ++k)
    if (k < p) out[2 + k] = a[k];
}

// The pairs' statistics from their sums, one thread per pair (the p-value's
// continued fraction is most of the work and does not fill a warp per pair). where
// (optional): the place of pair w in out. again (optional): collects the pairs whose
// S has lost more than kQgCancel of gg. Both kernels, n = 2000, p = 1, 54,600
// pairs: 0.94 -> 0.45 ms.
constexpr double kQgCancel = 1.0 / 1024;
__global__ void lmm_pair_stats_kernel(const double* __restrict__ sums, const int2* __restrict__ pairs, PairRange pr,
                                      int p, const double* __restrict__ chi0, const double* __restrict__ a00L,
                                      const double* __restrict__ rss, double df, const int* __restrict__ where,
                                      int* __restrict__ again, unsigned* __restrict__ n_again,
                                      eqtl_pair* __restrict__ out) {
  const int w = pr.first + blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= pr.end) return;
  const int g = pairs[w].x;
  const double* s = sums + static_cast<int64_t>(w - pr.first) * (p + 2);
  eqtl_pair q;
  q.snp = pairs[w].y;
  q.gene = g;
  q.reserved = 0;
  double S;
  lmm_stats_fp64(s[0], s[1], s + 2, chi0 + static_cast<int64_t>(g) * p, a00L + static_cast<int64_t>(g) * p * p, rss[g],
                 p, df, q, &S);
  out[where ? where[w] : w] = q;
  if (again && S < kQgCancel * s[0]) again[atomicAdd(n_again, 1u)] = w;
}

// ------------------------------------------------- tiny-|t| pairs in FP64
// Pairs screened with 0 < |t| < tiny_t need an FP64 t only to place them
// against the reference's x = df / (df + t^2) quantisation and to form their
// ACAT term; relative accuracy ~1e-8 is ample. So instead of rotating their
// raw dosages (n^2 per SNP):
//   NUM = g_raw . u,   u = Q (w o r~) for the gene (one DGEMM per scan),
//   S   = Gt'W Gt - a'A00^-1 a from the stored FP16 hi/lo rotated genotypes
//         (centred; S does not see the centring) accumulated in FP64.
__global__ void lmm_wr_kernel(const double* __restrict__ Ytil, const double* __restrict__ Xtil,
                              const double* __restrict__ lam, const double* __restrict__ delta,
                              const double* __restrict__ chi0, int n, int p, int G, double* wr) {
  const int g = blockIdx.x;
  if (g >= G) return;
  const double d = delta[g];
  const double* yt = Ytil + static_cast<int64_t>(g) * n;
  const double* c0 = chi0 + static_cast<int64_t>(g) * p;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double v = d * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    double r = yt[i];
    for (int k = 0; k < p; ++k) r -= Xtil[static_cast<int64_t>(k) * n + i] * c0[k];
    wr[static_cast<int64_t>(g) * n + i] = r / v;
  }
}

// Sums [num, gg, a_0 .. a_{p-1}] by a warp per pair, then p by a thread per pair, as
// for the refined pairs. n = 2000, p = 1, 62,000 pairs: 1.00 -> 0.65 ms.
template <int PM>
__global__ void lmm_tiny_sums_kernel(GenoRows src, const int32_t* __restrict__ col, int n, int k_pad,
                                     const int64_t* __restrict__ kept, const double* __restrict__ mu,
                                     const double* __restrict__ U, int64_t u_stride, const __half* __restrict__ gt_hi,
                                     const __half* __restrict__ gt_lo, double inv_s1, const double* __restrict__ Xtil,
                                     int p, const double* __restrict__ lam, const double* __restrict__ delta,
                                     const int2* __restrict__ pairs, PairRange pr, double* __restrict__ sums) {
  const int lane = threadIdx.x & 31;
  const int w = pr.first + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= pr.end) return;
  const int g = pairs[w].x;
  const int64_t r = pairs[w].y;
  const int64_t s = kept[r];
  const double mus = mu[s];
  const double* u = U + static_cast<int64_t>(g) * u_stride;
  const __half* gh = gt_hi + r * k_pad;
  const __half* gl = gt_lo + r * k_pad;
  const double d = delta[g];
  double num = 0, gg = 0, a[PM];
#pragma unroll
  for (int k = 0; k < PM; ++k) a[k] = 0;
#pragma unroll(PM <= 4 ? 8 : 2)
  for (int i = lane; i < n; i += 32) {
    const double dose = src.dosage(s, col[i]);
    num += (isnan(dose) ? mus : dose) * u[i];
    double v = d * lam[i] + 1.0;
    if (v < 1e-12) v = 1e-12;
    const double gt = (static_cast<double>(__half2float(gh[i])) + static_cast<double>(__half2float(gl[i]))) * inv_s1;
    const double dg = gt / v;
    gg += dg * gt;
#pragma unroll
    for (int k = 0; k < PM; ++k)
      if (k < p) a[k] += Xtil[static_cast<int64_t>(k) * n + i] * dg;
  }
  for (int o = 16; o; o >>= 1) {
    num += __shfl_xor_sync(0xffffffffu, num, o);
    gg += __shfl_xor_sync(0xffffffffu, gg, o);
#pragma unroll
    for (int k = 0; k < PM; ++k)
      if (k < p) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
  }
  if (lane != 0) return;
  double* out = sums + static_cast<int64_t>(w - pr.first) * (p + 2);
  out[0] = num;
  out[1] = gg;
#pragma unroll
  for (int k = 0; k < PM; ++k)
    if (k < p) out[2 + k] = a[k];
}
__global__ void lmm_tiny_p_kernel(const double* __restrict__ sums, const int2* __restrict__ pairs, PairRange pr, int p,
                                  const double* __restrict__ ainv, const double* __restrict__ rss, double df,
                                  double* __restrict__ p_out) {
  const int w = pr.first + blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= pr.end) return;
  const int g = pairs[w].x;
  const double* s = sums + static_cast<int64_t>(w - pr.first) * (p + 2);
  const double gg = s[1], *a = s + 2;
  eqtl_pair q;
  double S = -1.0;
  if (!(gg < 1e-12)) {
    const double* A = ainv + static_cast<int64_t>(g) * p * p;
    double aTu = 0;
    for (int x = 0; x < p; ++x) {
      double ux = 0;
      for (int y = 0; y < p; ++y) ux += A[x * p + y] * a[y];
      aTu += a[x] * ux;
    }
    S = gg - aTu;
  }
  lmm_stats_num_s(s[0], S, rss[g], df, q);
  p_out[w] = q.p;
}

}  // namespace dev

template <>
struct EpiOf<dev::RotEpiParams> {
  using type = dev::RotEpi;
};
template <>
struct EpiOf<dev::QgEpiParams> {
  using type = dev::QgEpi;
};
template <>
struct EpiOf<dev::LmmEpiParams<1>> {
  using type = dev::LmmEpi<1>;
};
template <>
struct EpiOf<dev::LmmEpiParams<2>> {
  using type = dev::LmmEpi<2>;
};
template <>
struct EpiOf<dev::LmmRawEpiParams<1>> {
  using type = dev::LmmEpi<1, false, true>;
};
template <>
struct EpiOf<dev::LmmLrEpiParams<1>> {
  using type = dev::LmmEpi<1, false, true, true>;
};
template <>
struct EpiOf<dev::LmmLrEpiParams<2>> {
  using type = dev::LmmEpi<2, false, true, true>;
};
template <>
struct EpiOf<dev::LmmNodeEpiParams<1>> {
  using type = dev::LmmNodeEpi<1>;
};
template <>
struct EpiOf<dev::LmmNodeEpiParams<2>> {
  using type = dev::LmmNodeEpi<2>;
};
template <>
struct EpiOf<dev::LmmRawEpiParams<2>> {
  using type = dev::LmmEpi<2, false, true>;
};
template <>
struct EpiOf<dev::LmmGroupEpiParams> {
  using type = dev::LmmGroupEpi;
};
template <>
struct EpiOf<dev::GlmEpiParams<1>> {
  using type = dev::LmmEpi<1, true>;
};
template <>
struct EpiOf<dev::GlmEpiParams<2>> {
  using type = dev::LmmEpi<2, true>;
};
template <>
struct EpiOf<dev::GlmGroupEpiParams> {
  using type = dev::GlmGroupEpi;
};

using namespace dev;

static cublasHandle_t blas_of(eqtl_ctx* ctx) {
  if (!ctx->cublas) {
    cublasHandle_t h;
    EQTL_CHECK(cublasCreate(&h) == CUBLAS_STATUS_SUCCESS, EQTL_E_CUDA, "cublasCreate failed");
    cublasSetStream(h, ctx->stream);
    ctx->cublas = h;
  }
  return static_cast<cublasHandle_t>(ctx->cublas);
}

// ------------------------------------------------------------------ basis
// --fast (sparsify_grm, src/model_lmm.cpp:88-104): off-diagonal entries of K
// below `thr` in magnitude become 0; the count of zeroed entries goes to *zeroed.
__global__ void sparsify_kernel(double* K, int n, double thr, unsigned long long* zeroed) {
  const int64_t total = static_cast<int64_t>(n) * n;
  unsigned long long c = 0;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i = e / n, j = e - i * n;
    if (i != j && fabs(K[e]) < thr) {
      K[e] = 0.0;
      ++c;
    }
  }
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(zeroed, c);
}

void lmm_basis_from_grm(eqtl_ctx* ctx, const double* K_dev, int n, double sparsify_thr, int64_t* zeroed) {
  cudaStream_t st = ctx->stream;
  StageScope timer(ctx, EQTL_STAGE_EIGEN);
  LmmBasisDev& B = ctx->basis;
  B.n = n;
  B.Q.alloc(static_cast<size_t>(n) * n);
  B.lambda.alloc(n);
  EQTL_CUDA(cudaMemcpyAsync(B.Q.p, K_dev, sizeof(double) * n * n, cudaMemcpyDeviceToDevice, st));
  if (sparsify_thr > 0) {
    DevBuf<unsigned long long>& cnt = ctx->ws.sparsify_cnt;
    cnt.alloc(1);
    cnt.zero(st);
    ++ctx->launches;
    const int64_t total = static_cast<int64_t>(n) * n;
    sparsify_kernel<<<static_cast<unsigned>(std::min<int64_t>((total + 255) / 256, 1184)), 256, 0, st>>>(
        B.Q.p, n, sparsify_thr, cnt.p);
    EQTL_CUDA(cudaGetLastError());
    unsigned long long c = 0;
    cnt.download(&c, 1, st);
    EQTL_CUDA(cudaStreamSynchronize(st));
    if (zeroed) *zeroed = static_cast<int64_t>(c);
  }
  if (!ctx->cusolver) {
    cusolverDnHandle_t hc;
    EQTL_CHECK(cusolverDnCreate(&hc) == CUSOLVER_STATUS_SUCCESS, EQTL_E_CUDA, "cusolverDnCreate failed");
    ctx->cusolver = hc;
  }
  cusolverDnHandle_t h = static_cast<cusolverDnHandle_t>(ctx->cusolver);
  cusolverDnSetStream(h, st);
  int lwork = 0;
  cusolverStatus_t cs = cusolverDnDsyevd_bufferSize(h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, n, B.Q.p, n,
                                                    B.lambda.p, &lwork);
  DevBuf<double>& work = ctx->ws.eig_work;
  DevBuf<int>& info = ctx->ws.eig_info;
  if (cs == CUSOLVER_STATUS_SUCCESS) {
    work.alloc(std::max(lwork, 1));
    info.alloc(1);
    cs = cusolverDnDsyevd(h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, n, B.Q.p, n, B.lambda.p, work.p, lwork,
                          info.p);
  }
  int info_h = 0;
  if (cs == CUSOLVER_STATUS_SUCCESS) {
    info.download(&info_h, 1, st);
    EQTL_CUDA(cudaStreamSynchronize(st));
  }
  EQTL_CHECK(cs == CUSOLVER_STATUS_SUCCESS && info_h == 0, EQTL_E_CUDA, "GRM eigen decomposition failed");
  B.lambda_h.resize(n);
  B.lambda.download(B.lambda_h.data(), n, st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  for (double& l : B.lambda_h) l = std::max(l, 0.0);  // cwiseMax(0.0)
  B.lambda.upload(B.lambda_h.data(), n, st);
  B.Q_h.clear();
  B.sliced = false;
  ctx->have_basis = true;
  ctx->rot.m = 0;  // rotated genotypes belong to the previous basis
}

void solver_release(eqtl_ctx* ctx) {
  if (ctx->cusolver) cusolverDnDestroy(static_cast<cusolverDnHandle_t>(ctx->cusolver));
  ctx->cusolver = nullptr;
}

void lmm_set_basis(eqtl_ctx* ctx, const double* Q, const double* lambda, int n) {
  LmmBasisDev& B = ctx->basis;
  B.n = n;
  B.Q.upload(Q, static_cast<size_t>(n) * n, ctx->stream);
  B.lambda_h.assign(lambda, lambda + n);
  for (double& l : B.lambda_h) l = std::max(l, 0.0);
  B.lambda.upload(B.lambda_h.data(), n, ctx->stream);
  EQTL_CUDA(cudaStreamSynchronize(ctx->stream));
  B.sliced = false;
  ctx->have_basis = true;
  ctx->rot.m = 0;
}

// --------------------------------------------------------------- rotation
static void output_scales(int n, float& s1, float& s2) {
  // |Gt| <= |g - mean|_2 <= 2 sqrt(n); |Gt^2| <= 4 n: keep both below ~3e4
  s1 = std::ldexp(1.0f, static_cast<int>(std::floor(std::log2(30000.0 / (2.0 * std::sqrt(static_cast<double>(n)))))));
  s2 = std::ldexp(1.0f, static_cast<int>(std::floor(std::log2(30000.0 / (4.0 * n)))));
}

void lmm_rotate(eqtl_ctx* ctx) {
  Geno& g = ctx->geno;
  Rotated& R = ctx->rot;
  EQTL_CHECK(ctx->have_basis && ctx->basis.n == g.n, EQTL_E_STATE, "rotation needs an eigenbasis of size n");
  if (R.m == g.m && R.k_pad == g.k_pad && R.gt_hi.p) return;
  R.bf16_m = -1;
  cudaStream_t st = ctx->stream;
  StageScope timer(ctx, EQTL_STAGE_ROTATE);
  const int n = g.n, k_pad = g.k_pad;
  const int64_t m = g.m;
  DevBuf<__half>& qh = ctx->ws.q_hi;
  DevBuf<__half>& ql = ctx->ws.q_lo;
  ++ctx->launches;
  qh.alloc(static_cast<size_t>(n) * k_pad);
  ql.alloc(static_cast<size_t>(n) * k_pad);
  // split-BF16 contexts hold the genotype operand in BF16, so Q' is split
  // in BF16 too and the rotation runs on BF16 pairs
  const bool bf16 = ctx->precision == EQTL_PREC_SPLIT_BF16;
  if (bf16)
    q_split_kernel<__nv_bfloat16><<<dim3((k_pad + 255) / 256, n), 256, 0, st>>>(
        ctx->basis.Q.p, n, k_pad, reinterpret_cast<__nv_bfloat16*>(qh.p), reinterpret_cast<__nv_bfloat16*>(ql.p));
  else
    q_split_kernel<__half><<<dim3((k_pad + 255) / 256, n), 256, 0, st>>>(ctx->basis.Q.p, n, k_pad, qh.p, ql.p);
  EQTL_CUDA(cudaGetLastError());
  const size_t elems = static_cast<size_t>(m) * k_pad;
  R.gt_hi.alloc(elems);
  R.gt_lo.alloc(elems);
  R.gt2_hi.alloc(elems);
  R.gt2_lo.alloc(elems);
  // The epilogue's 128-row tiles reach past k_pad (a multiple of 64), so it writes
  // the zero columns from n on too: clearing the four operands first took 1.25 of
  // 9.9 ms (n = 2000, 5e5 SNPs).
  RotEpiParams ep{};
  ep.m = m;
  ep.k_pad = k_pad;
  ep.unscale = 1.0f / (kGcScale * 1024.0f);
  output_scales(n, ep.s1, ep.s2);
  ep.gt_hi = R.gt_hi.p;
  ep.gt_lo = R.gt_lo.p;
  ep.gt2_hi = R.gt2_hi.p;
  ep.gt2_lo = R.gt2_lo.p;
  if (m > 0) {
    const __half* ah[1] = {qh.p};
    const __half* al[1] = {ql.p};
    const __half* bh[1] = {g.gc_hi.p};
    const __half* bl[1] = {g.gc_lo.p};
    const int bsel[1] = {0}, prod[1] = {7};
    if (!bf16 && tile_pairs(n))
      launch_tile_n<256, 1, RotEpiParams, dev::kBLoStage, 2>(ctx, false, ep, ah, al, n, bh, bl, m, k_pad, bsel, prod);
    else
      launch_tile_n<256, 1>(ctx, bf16, ep, ah, al, n, bh, bl, m, k_pad, bsel, prod);
  }
  if (ctx->precision == EQTL_PREC_FP32_SIMT && m > 0) {
    // the FP32 form keeps its SNP-side operands in FP32
    R.gt32.alloc(elems);
    R.gt2_32.alloc(elems);
    ctx->launches += 2;
    sum_split_kernel<<<1184, 256, 0, st>>>(R.gt_hi.p, R.gt_lo.p, static_cast<int64_t>(elems), R.gt32.p);
    sum_split_kernel<<<1184, 256, 0, st>>>(R.gt2_hi.p, R.gt2_lo.p, static_cast<int64_t>(elems), R.gt2_32.p);
    EQTL_CUDA(cudaGetLastError());
  }
  R.m = m;
  R.k_pad = k_pad;
}

// ------------------------------------------------------------------- REML
// Per-gene REML prep into the context workspace (ws.Ytil, Xtil, delta, chi0,
// ainv, rss) from the resident phenotypes.
// out[i] = x[i]^2
__global__ void square_kernel(const double* __restrict__ x, int64_t count, double* out) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = x[i] * x[i];
}

// Batched REML for p > kRemlWarpP over ws.Ytil / ws.Xtil into ws.delta,
// chi0, ainv, rss: columns in chunks whose per-round buffers stay near 2 GB.
template <int GW>
static void reml_batched(eqtl_ctx* ctx, int n, int p, int G) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  cublasHandle_t h = blas_of(ctx);
  const int nq = p * (p + 1) / 2;
  const int df = n - p;
  ws.rb_P.alloc(static_cast<size_t>(nq) * n);
  ++ctx->launches;
  rb_pairs_kernel<<<1184, 256, 0, st>>>(ws.Xtil.p, n, p, ws.rb_P.p);
  EQTL_CUDA(cudaGetLastError());
  // grid-phase quantities shared by every column
  {
    const int K = kRbGridN;
    ws.rb_Wg.alloc(static_cast<size_t>(n) * K);
    ws.rb_Xw.alloc(static_cast<size_t>(n) * K * p);
    ws.rb_Ag.alloc(static_cast<size_t>(nq) * K);
    ws.rb_Lg.alloc(static_cast<size_t>(K) * p * p);
    ws.rb_ldx.alloc(K);
    ws.rb_ldD.alloc(K);
    ctx->launches += 2;
    rb_grid_weights_kernel<<<K, 256, 0, st>>>(ws.Xtil.p, ctx->basis.lambda.p, n, p, ws.rb_Wg.p, ws.rb_Xw.p,
                                             ws.rb_ldD.p);
    EQTL_CUDA(cudaGetLastError());
    const double one = 1.0, zero = 0.0;
    EQTL_CHECK(cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, nq, K, n, &one, ws.rb_P.p, nq, ws.rb_Wg.p, n, &zero,
                           ws.rb_Ag.p, nq) == CUBLAS_STATUS_SUCCESS,
               EQTL_E_CUDA, "REML grid X'DX failed");
    rb_grid_chol_kernel<GW><<<(K * GW + 127) / 128, 128, 0, st>>>(ws.rb_Ag.p, p, ws.rb_Lg.p, ws.rb_ldx.p);
    EQTL_CUDA(cudaGetLastError());
  }
  const int cmax = std::max(1024, static_cast<int>((int64_t(1) << 26) / std::max(n, 1)));
  for (int g0 = 0; g0 < G; g0 += cmax) {
    const int C = std::min(cmax, G - g0);
    const size_t slots = 2 * static_cast<size_t>(C);
    ws.rb_state.alloc(sizeof(RemlBatchState) * C);
    ws.rb_dlt.alloc(slots);
    ws.rb_W.alloc(slots * n);
    ws.rb_WY.alloc(slots * n);
    ws.rb_A.alloc(slots * nq);
    ws.rb_B.alloc(slots * p);
    ws.rb_ld.alloc(slots);
    ws.rb_ydy.alloc(slots);
    ws.rb_active.alloc(1);
    RemlBatchState* state = reinterpret_cast<RemlBatchState*>(ws.rb_state.p);
    const double* Y = ws.Ytil.p + static_cast<int64_t>(g0) * n;
    const unsigned cblocks = static_cast<unsigned>((C + 127) / 128);
    const double one = 1.0, zero = 0.0;
    // grid phase: X~'D_k y for all columns as one GEMM over the stacked
    // w_k o X~ (35 p rows), y'D_k y as one GEMM over y o y
    {
      const int K = kRbGridN;
      ws.rb_Bg.alloc(static_cast<size_t>(K) * p * C);
      ws.rb_Yg.alloc(static_cast<size_t>(K) * C);
      ctx->launches += 1;
      square_kernel<<<1184, 256, 0, st>>>(Y, static_cast<int64_t>(n) * C, ws.rb_WY.p);
      EQTL_CUDA(cudaGetLastError());
      EQTL_CHECK(cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, K * p, C, n, &one, ws.rb_Xw.p, n, Y, n, &zero,
                             ws.rb_Bg.p, K * p) == CUBLAS_STATUS_SUCCESS,
                 EQTL_E_CUDA, "REML grid X'Dy failed");
      EQTL_CHECK(cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, K, C, n, &one, ws.rb_Wg.p, n, ws.rb_WY.p, n, &zero,
                             ws.rb_Yg.p, K) == CUBLAS_STATUS_SUCCESS,
                 EQTL_E_CUDA, "REML grid y'Dy failed");
      ctx->launches += 2;
      ws.rb_V.alloc(static_cast<size_t>(K) * C);
      rb_grid_eval_kernel<GW><<<dim3(cblocks, K), 128, 0, st>>>(C, p, df, ws.rb_Lg.p, ws.rb_ldx.p, ws.rb_ldD.p,
                                                                 ws.rb_Bg.p, ws.rb_Yg.p, ws.rb_V.p);
      rb_grid_advance_kernel<<<cblocks, 128, 0, st>>>(C, df, ws.rb_V.p, state, ws.rb_dlt.p);
      EQTL_CUDA(cudaGetLastError());
    }
    // the sums of every slot's delta
    auto sums = [&] {
      ++ctx->launches;
      rb_weights_kernel<<<static_cast<unsigned>((slots + 7) / 8), 256, 0, st>>>(
          Y, ctx->basis.lambda.p, n, C, ws.rb_dlt.p, ws.rb_W.p, ws.rb_WY.p, ws.rb_ld.p, ws.rb_ydy.p);
      EQTL_CUDA(cudaGetLastError());
      EQTL_CHECK(cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, nq, static_cast<int>(slots), n, &one, ws.rb_P.p, nq,
                             ws.rb_W.p, n, &zero, ws.rb_A.p, nq) == CUBLAS_STATUS_SUCCESS,
                 EQTL_E_CUDA, "REML X'DX failed");
      EQTL_CHECK(cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, p, static_cast<int>(slots), n, &one, ws.Xtil.p, n,
                             ws.rb_WY.p, n, &zero, ws.rb_B.p, p) == CUBLAS_STATUS_SUCCESS,
                 EQTL_E_CUDA, "REML X'Dy failed");
    };
    // the golden phase runs the same number of rounds for every column; from
    // the Newton phase on, stop once no column is left searching
    for (int round = 0; df > 0 && round < kRbMaxRounds - 1; ++round) {
      sums();
      ++ctx->launches;
      EQTL_CUDA(cudaMemsetAsync(ws.rb_active.p, 0, sizeof(unsigned int), st));
      constexpr int kCols = kRbThreads / GW / 2;
      rb_advance_kernel<GW><<<static_cast<unsigned>((C + kCols - 1) / kCols), kRbThreads, 0, st>>>(
          C, p, df, ws.rb_A.p, ws.rb_B.p, ws.rb_ld.p, ws.rb_ydy.p, state, ws.rb_dlt.p, ws.rb_active.p);
      EQTL_CUDA(cudaGetLastError());
      if (round >= 40) {
        unsigned int left = 0;
        ws.rb_active.download(&left, 1, st);
        EQTL_CUDA(cudaStreamSynchronize(st));
        if (left == 0) break;
      }
    }
    sums();
    ++ctx->launches;
    constexpr int kGroups = kRbThreads / GW;
    rb_final_kernel<GW><<<static_cast<unsigned>((C + kGroups - 1) / kGroups), kRbThreads, 0, st>>>(
        C, g0, p, ws.rb_A.p, ws.rb_B.p, ws.rb_ydy.p, state, ws.delta.p, ws.chi0.p, ws.ainv.p, ws.rss.p, ws.a00L.p);
    EQTL_CUDA(cudaGetLastError());
  }
}

void lmm_prep(eqtl_ctx* ctx, const PhenoDev& ph, bool y_rotated) {
  const int n = ph.n, G = ph.G, p = ph.p;
  EQTL_CHECK(ctx->have_basis && ctx->basis.n == n, EQTL_E_STATE, "LMM prep needs an eigenbasis of size n");
  EQTL_CHECK(p >= 1 && p <= kMaxPLmm, EQTL_E_UNSUPPORTED, "the device LMM handles 1 <= p <= 32 covariate columns");
  cudaStream_t st = ctx->stream;
  Workspace& ws = ctx->ws;
  cublasHandle_t h = blas_of(ctx);
  ws.Ytil.alloc(static_cast<size_t>(n) * G);
  ws.Xtil.alloc(static_cast<size_t>(n) * p);
  const double one = 1.0, zero = 0.0;
  if (y_rotated) {
    EQTL_CUDA(cudaMemcpyAsync(ws.Ytil.p, ph.Y.p, sizeof(double) * n * G, cudaMemcpyDeviceToDevice, st));
  } else {
    EQTL_CHECK(cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, n, G, n, &one, ctx->basis.Q.p, n, ph.Y.p, n, &zero,
                           ws.Ytil.p, n) == CUBLAS_STATUS_SUCCESS,
               EQTL_E_CUDA, "Q'Y failed");
  }
  EQTL_CHECK(cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, n, p, n, &one, ctx->basis.Q.p, n, ph.X.p, n, &zero, ws.Xtil.p,
                         n) == CUBLAS_STATUS_SUCCESS,
             EQTL_E_CUDA, "Q'X failed");
  ws.delta.alloc(G);
  ws.chi0.alloc(static_cast<size_t>(G) * p);
  ws.ainv.alloc(static_cast<size_t>(G) * p * p);
  ws.a00L.alloc(static_cast<size_t>(G) * p * p);
  ws.rss.alloc(G);
  if (p <= kRemlWarpP) {
    ws.reml_w.alloc(static_cast<size_t>(kRbGridN) * n);
    ws.reml_tot.alloc(static_cast<size_t>(kRbGridN) * (1 + p * (p + 1) / 2));
    ctx->launches += 2;
    auto run = [&](auto pc) {
      constexpr int P = decltype(pc)::value;
      reml_grid_kernel<P><<<kRbGridN, 32, 0, st>>>(ws.Xtil.p, ctx->basis.lambda.p, n, ws.reml_w.p, ws.reml_tot.p);
      constexpr int per = kRemlThreads / 32;
      reml_warp_kernel<P><<<static_cast<unsigned>((G + per - 1) / per), kRemlThreads, 0, st>>>(
          ws.Ytil.p, ws.Xtil.p, ctx->basis.lambda.p, n, G, ws.reml_w.p, ws.reml_tot.p, ws.delta.p, ws.chi0.p,
          ws.ainv.p, ws.rss.p, ws.a00L.p);
    };
    if (p == 1) run(std::integral_constant<int, 1>{});
    else if (p == 2) run(std::integral_constant<int, 2>{});
    else run(std::integral_constant<int, 3>{});
    EQTL_CUDA(cudaGetLastError());
    return;
  }
  ++ctx->launches;
  // lanes per factorisation: the smallest group that holds p rows
  if (p <= 8) reml_batched<8>(ctx, n, p, G);
  else if (p <= 16) reml_batched<16>(ctx, n, p, G);
  else reml_batched<kMaxPLmm>(ctx, n, p, G);
}

// ------------------------------------------------------------------- scan
// hi + lo of an FP16 pair operand, re-split into BF16 hi + lo (the split-BF16
// form of the scans: ~16 significant bits instead of ~22)
__global__ void resplit_bf16_kernel(const __half* __restrict__ hi, const __half* __restrict__ lo, int64_t count,
                                    __nv_bfloat16* bhi, __nv_bfloat16* blo) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float v = __half2float(hi[i]) + __half2float(lo[i]);
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    bhi[i] = h;
    blo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
  }
}

static void resplit_bf16(eqtl_ctx* ctx, const __half* hi, const __half* lo, int64_t count, DevBuf<__half>& bhi,
                         DevBuf<__half>& blo) {
  bhi.alloc(static_cast<size_t>(std::max<int64_t>(count, 1)));
  blo.alloc(static_cast<size_t>(std::max<int64_t>(count, 1)));
  if (count <= 0) return;
  ++ctx->launches;
  resplit_bf16_kernel<<<static_cast<unsigned>(std::min<int64_t>((count + 255) / 256, int64_t(ctx->sm_count) * 32)),
                        256, 0, ctx->stream>>>(hi, lo, count, reinterpret_cast<__nv_bfloat16*>(bhi.p),
                                               reinterpret_cast<__nv_bfloat16*>(blo.p));
  EQTL_CUDA(cudaGetLastError());
}

// The split-BF16 SNP-side operands of the rotation (once per rotation).
static void rot_bf16(eqtl_ctx* ctx, Rotated& R) {
  if (R.bf16_m == R.m && R.bgt_hi.p) return;
  const int64_t elems = R.m * R.k_pad;
  resplit_bf16(ctx, R.gt_hi.p, R.gt_lo.p, elems, R.bgt_hi, R.bgt_lo);
  resplit_bf16(ctx, R.gt2_hi.p, R.gt2_lo.p, elems, R.bgt2_hi, R.bgt2_lo);
  R.bf16_m = R.m;
}

// The split-BF16 gene-side operands: nops pairs of rows x k_pad into
// ws.opsb_hi / opsb_lo; out[j], out[nops + j] point at pair j's hi and lo.
static void gene_ops_bf16(eqtl_ctx* ctx, const __half* const* hi, const __half* const* lo, int nops, int64_t rows,
                          int k_pad, const __half** out) {
  EQTL_CHECK(nops <= dev::kMaxAcc, EQTL_E_INTERNAL, "split-BF16 gene operands");
  for (int j = 0; j < nops; ++j) {
    resplit_bf16(ctx, hi[j], lo[j], rows * k_pad, ctx->ws.opsb_hi[j], ctx->ws.opsb_lo[j]);
    out[j] = ctx->ws.opsb_hi[j].p;
    out[nops + j] = ctx->ws.opsb_lo[j].p;
  }
}

template <int P>
static void lmm_launch_simt(eqtl_ctx* ctx, const LmmEpiParams<P>& ep, const __half* const* ah,
                            const __half* const* al, int G, const __half* const* bh, const __half* const* bl,
                            const int* bsel, const Rotated& R);

// Gene-ops index (0 NUM, 1 .. p a_k, p + 1 gg) of the tile's accumulator j
// (LmmEpi): [NUM, gg, a_0] on the tensor cores with p = 1, else [gg, a_0 .., NUM].
static int lmm_acc_op(int p, int j, bool tensor) {
  if (tensor && p == 1) return j == 0 ? 0 : (j == 1 ? 2 : 1);
  return j == 0 ? p + 1 : (j == p + 1 ? 0 : j);
}

template <int P, class EP>
static void lmm_launch(eqtl_ctx* ctx, const EP& ep, const __half* const* ah, const __half* const* al, int G,
                       bool simt, const int2* tiles, int n_tiles, const Rotated& R) {
  // the exact-operand form reads the raw SNP operand (one exact FP16 slice:
  // hi*hi + lo*hi) for NUM and a_k, and Gt^2 for gg as both forms do
  constexpr bool raw = std::is_same_v<EP, LmmRawEpiParams<P>>;
  const __half* bh[2] = {raw ? R.raw.p : R.gt_hi.p, R.gt2_hi.p};
  const __half* bl[2] = {raw ? R.raw.p : R.gt_lo.p, R.gt2_lo.p};
  // the tile's accumulators [NUM, gg, a_0] (p = 1, tensor cores) or [gg, a_0 ..
  // a_{P-1}, NUM] from the gene-ops order [NUM, a.., gg]
  const __half* oh[P + 2];
  const __half* ol[P + 2];
  int bsel[P + 2], prod[P + 2];
  for (int j = 0; j < P + 2; ++j) {
    const int op = lmm_acc_op(P, j, !simt);
    oh[j] = ah[op];
    ol[j] = al[op];
    bsel[j] = op == P + 1 ? 1 : 0;  // gg reads Gt^2
    prod[j] = raw && op != P + 1 ? 5 : 7;
  }
  ah = oh;
  al = ol;
  if (!simt && !raw && ctx->precision == EQTL_PREC_SPLIT_BF16) {
    // split-BF16: both sides re-split into BF16 hi + lo, three products each
    const __half* b16[2 * (P + 2)];
    gene_ops_bf16(ctx, ah, al, P + 2, G, R.k_pad, b16);
    Rotated& Rw = const_cast<Rotated&>(R);
    rot_bf16(ctx, Rw);
    const __half* sbh[2] = {Rw.bgt_hi.p, Rw.bgt2_hi.p};
    const __half* sbl[2] = {Rw.bgt_lo.p, Rw.bgt2_lo.p};
    launch_tile_n<128, P + 2>(ctx, true, ep, b16, b16 + (P + 2), G, sbh, sbl, R.m, R.k_pad, bsel, prod, tiles,
                              n_tiles);
    return;
  }
  if (!simt) {
    launch_tile_n<128, P + 2>(ctx, false, ep, ah, al, G, bh, bl, R.m, R.k_pad, bsel, prod, tiles, n_tiles);
    return;
  }
  if constexpr (std::is_same_v<EP, LmmEpiParams<P>>) lmm_launch_simt<P>(ctx, ep, ah, al, G, bh, bl, bsel, R);
}

// the plain FP32 CUDA-core comparator of the LMM scan
// The FP32 operands (ws.ops32 in tile order, Rotated::gt32 / gt2_32) are
// formed before the scan; accumulator 0 (gg) reads Gt^2, the others Gt.
template <int P>
static void lmm_launch_simt(eqtl_ctx* ctx, const LmmEpiParams<P>& ep, const __half* const*, const __half* const*,
                            int G, const __half* const*, const __half* const*, const int* bsel, const Rotated& R) {
  cudaStream_t st = ctx->stream;
  EQTL_CHECK(bsel[0] == 1 && R.gt32.p && R.gt2_32.p, EQTL_E_INTERNAL, "FP32 comparator operands");
  const float* ptrs[P + 2];
  for (int j = 0; j < P + 2; ++j) ptrs[j] = ctx->ws.ops32[j].p;
  DevBuf<const float*>& dptr = ctx->ws.ops32_ptr;
  dptr.upload(ptrs, P + 2, st);
  TileShape sh{};
  using Cfg = SimtCfg<P + 2>;
  auto kern = simt_tile_kernel<P + 2, LmmSimtEpi<P>>;
  EQTL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
  dim3 grid(static_cast<unsigned>((R.m + kSimtBN - 1) / kSimtBN), static_cast<unsigned>((G + kSimtBM - 1) / kSimtBM));
  ++ctx->launches;
  kern<<<grid, kSimtThreads, Cfg::SMEM_BYTES, st>>>(dptr.p, G, R.gt32.p, R.gt2_32.p, R.m, R.k_pad, sh, ep);
  EQTL_CUDA(cudaGetLastError());
  EQTL_CUDA(cudaStreamSynchronize(st));
}

// Q'g of the listed SNPs (snps; on the device in ws.ref_snps) from their exact
// dosages by the digits of Q, into out [u][n].
static void exact_qg(eqtl_ctx* ctx, const std::vector<int>& snps, double* out) {
  const Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  LmmBasisDev& B = ctx->basis;
  cudaStream_t st = ctx->stream;
  const int n = g.n, k_pad = g.k_pad, u = static_cast<int>(snps.size());
  const int64_t rows = qg_rows(n);
  if (!B.sliced) {
    B.digits.alloc(static_cast<size_t>(rows) * k_pad);
    B.digit_scale.alloc(static_cast<size_t>(n));
    B.digits.zero(st);  // the rows that hold no digit
    ++ctx->launches;
    q_digits_kernel<<<n, 256, 0, st>>>(B.Q.p, n, k_pad, B.digits.p, B.digit_scale.p);
    EQTL_CUDA(cudaGetLastError());
    B.sliced = true;
  }
  // (over the load's samples, of which a view has a part)
  const bool any_missing = std::any_of(snps.begin(), snps.end(), [&](int r) {
    return g.n_miss_h[static_cast<size_t>(g.kept_h[static_cast<size_t>(r)])] > 0;
  });
  ws.qg_dose.alloc(static_cast<size_t>(u) * k_pad);
  if (any_missing) ws.qg_mask.alloc(static_cast<size_t>(u) * k_pad);
  ++ctx->launches;
  listed_dosage_kernel<<<(u + 7) / 8, 256, 0, st>>>(g.rows(), g.col.p, n, k_pad, g.kept.p, ws.ref_snps.p, u,
                                                    ws.qg_dose.p, any_missing ? ws.qg_mask.p : nullptr);
  EQTL_CUDA(cudaGetLastError());
  QgEpiParams ep{n, u, B.digit_scale.p, nullptr, g.kept.p, ws.ref_snps.p, out};
  auto pass = [&](const __half* snp_side) {
    const __half* ap[1] = {B.digits.p};
    const __half* bp[1] = {snp_side};
    const int bsel[1] = {0}, prod[1] = {1};
    if (tile_pairs(rows))
      launch_tile_n<256, 1, QgEpiParams, dev::kBLoNone, 2>(ctx, false, ep, ap, ap, rows, bp, bp, u, k_pad, bsel, prod);
    else
      launch_tile_n<256, 1, QgEpiParams, dev::kBLoNone>(ctx, false, ep, ap, ap, rows, bp, bp, u, k_pad, bsel, prod);
  };
  pass(ws.qg_dose.p);
  if (any_missing) {
    ep.mu = g.mu.p;
    pass(ws.qg_mask.p);
  }
}

// f(std::integral_constant<int, PM>) with the least PM >= p of the per-pair kernels.
template <class F>
static void with_p(int p, F&& f) {
  if (p <= 2) f(std::integral_constant<int, 2>{});
  else if (p <= 4) f(std::integral_constant<int, 4>{});
  else if (p <= 8) f(std::integral_constant<int, 8>{});
  else if (p <= 16) f(std::integral_constant<int, 16>{});
  else f(std::integral_constant<int, kMaxPLmm>{});
}

// f(PairRange) over n_pairs pairs in pieces whose sums, `width` doubles a pair, take at
// most 32 MB of ws.ref_sums (a threshold near 1 refines every pair: 10^8 of them with
// ten covariates would take 10 GB).
template <class F>
static void by_sums(Workspace& ws, int n_pairs, int width, F&& f) {
  const int piece = std::min(n_pairs, (1 << 22) / width);
  ws.ref_sums.alloc(static_cast<size_t>(piece) * width);
  for (int first = 0; first < n_pairs; first += piece) f(PairRange{first, first + std::min(piece, n_pairs - first)});
}

// Gt = Q'g of the u listed SNPs (ws.ref_snps) into ws.gt by DGEMM, with `pad`
// zero columns after them.
static void dgemm_qg(eqtl_ctx* ctx, int u, int pad) {
  Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  const int n = g.n, cols = u + pad;
  ws.gt.alloc(static_cast<size_t>(n) * cols);
  ws.graw.alloc(static_cast<size_t>(n) * cols);
  ++ctx->launches;
  raw_dosage_kernel<<<1184, 256, 0, ctx->stream>>>(g.rows(), g.col.p, n, g.kept.p, g.mu.p, ws.ref_snps.p, u, ws.graw.p);
  EQTL_CUDA(cudaGetLastError());
  if (pad)
    EQTL_CUDA(cudaMemsetAsync(ws.graw.p + static_cast<size_t>(n) * u, 0, sizeof(double) * n * pad, ctx->stream));
  const double one = 1.0, zero = 0.0;
  EQTL_CHECK(cublasDgemm(blas_of(ctx), CUBLAS_OP_T, CUBLAS_OP_N, n, cols, n, &one, ctx->basis.Q.p, n, ws.graw.p, n,
                         &zero, ws.gt.p, n) == CUBLAS_STATUS_SUCCESS,
             EQTL_E_CUDA, "Q'g failed");
}

// FP64 statistics of the first n_pairs of ws.ref_pairs into ws.refined, against the
// current LMM prep (ws.Ytil, Xtil, delta, chi0, ainv, rss): Gt = Q'g of the SNPs
// involved (exactly on the tensor cores for many 2-bit rows, else by DGEMM: FP32
// dosages, more than kQgMaxN samples, little work), then the pairs' sums and
// statistics.
//
// A gene whose delta is at the top of its search leaves S = gg - a'A00^-1 a with a
// millionth of gg: its last digits are Q'g's rounding, and p moves by 1e-8 with the
// way Q'g was summed. Pairs of an exact list that lose more than kQgCancel so are done
// again by DGEMM over at least kQgDgemmCols columns, where its bits depended on the
// number of columns at one of ten n tried, so that two long lists agree about such a
// pair. A list below kQgMinWork takes the DGEMM of its own width, which sums in another
// order when it has few columns: there the pair keeps only what its S keeps.
static void lmm_refine_pairs(eqtl_ctx* ctx, int p, double df, int n_pairs) {
  Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  const int n = g.n;
  if (n_pairs == 0) return;
  const std::vector<int> snps = distinct_snps(ctx, ws.ref_pairs.p, n_pairs, g.m);
  const int u = static_cast<int>(snps.size());
  const bool exact = !g.dense && n <= kQgMaxN && static_cast<int64_t>(n) * n * u >= kQgMinWork;
  ws.refined.alloc(static_cast<size_t>(n_pairs));
  auto refine = [&](const int2* pairs, int count, const int* where, int* again, unsigned* n_again) {
    by_sums(ws, count, p + 2, [&](PairRange pr) {
      const int k = pr.end - pr.first;
      ctx->launches += 2;
      with_p(p, [&](auto pm) {
        lmm_pair_sums_kernel<decltype(pm)::value><<<static_cast<unsigned>((k + 7) / 8), 256, 0, st>>>(
            ws.gt.p, n, ws.ref_col.p, pairs, pr, ws.Ytil.p, ws.Xtil.p, p, ctx->basis.lambda.p, ws.delta.p,
            ws.ref_sums.p);
      });
      lmm_pair_stats_kernel<<<static_cast<unsigned>((k + 63) / 64), 64, 0, st>>>(
          ws.ref_sums.p, pairs, pr, p, ws.chi0.p, ws.a00L.p, ws.rss.p, df, where, again, n_again, ws.refined.p);
      EQTL_CUDA(cudaGetLastError());
    });
  };
  if (!exact) {
    dgemm_qg(ctx, u, 0);
    refine(ws.ref_pairs.p, n_pairs, nullptr, nullptr, nullptr);
    return;
  }
  ws.gt.alloc(static_cast<size_t>(n) * u);
  exact_qg(ctx, snps, ws.gt.p);
  ws.ref_again.alloc(static_cast<size_t>(n_pairs));
  ws.ref_n_again.alloc(1);
  ws.ref_n_again.zero(st);
  refine(ws.ref_pairs.p, n_pairs, nullptr, ws.ref_again.p, ws.ref_n_again.p);
  unsigned n_again = 0;
  ws.ref_n_again.download(&n_again, 1, st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  if (n_again == 0) return;
  ws.pairs_again.alloc(n_again);
  ++ctx->launches;
  listed_pairs_kernel<<<(n_again + 255) / 256, 256, 0, st>>>(ws.ref_pairs.p, ws.ref_again.p,
                                                             static_cast<int>(n_again), ws.pairs_again.p);
  EQTL_CUDA(cudaGetLastError());
  const int v = static_cast<int>(distinct_snps(ctx, ws.pairs_again.p, static_cast<int>(n_again), g.m).size());
  dgemm_qg(ctx, v, std::max(0, kQgDgemmCols - v));
  refine(ws.pairs_again.p, static_cast<int>(n_again), ws.ref_again.p, nullptr, nullptr);
}

// FP64 p of the n_tiny pairs of ws.tiny_pairs against the current LMM prep (see
// lmm_tiny_sums_kernel).
// U_pre (optional): u = Q (w o r~) of gene g at U_pre + g * u_stride, as the
// exact-operand scan has it already; otherwise it is computed here.
static std::vector<double> lmm_tiny_p(eqtl_ctx* ctx, int p, double df, int n_tiny,
                                      const double* U_pre = nullptr, int64_t u_stride = 0) {
  Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  Rotated& R = ctx->rot;
  cudaStream_t st = ctx->stream;
  const int n = g.n;
  const int G = static_cast<int>(ws.delta.n);
  std::vector<double> out(static_cast<size_t>(n_tiny));
  if (n_tiny == 0) return out;
  const double* U = U_pre;
  if (!U) {
    ws.graw.alloc(static_cast<size_t>(n) * G);  // w o r~ per gene
    ws.gt.alloc(static_cast<size_t>(n) * G);    // u = Q (w o r~)
    ctx->launches += 1;
    lmm_wr_kernel<<<G, 256, 0, st>>>(ws.Ytil.p, ws.Xtil.p, ctx->basis.lambda.p, ws.delta.p, ws.chi0.p, n, p, G,
                                     ws.graw.p);
    EQTL_CUDA(cudaGetLastError());
    const double one = 1.0, zero = 0.0;
    EQTL_CHECK(cublasDgemm(blas_of(ctx), CUBLAS_OP_N, CUBLAS_OP_N, n, G, n, &one, ctx->basis.Q.p, n, ws.graw.p, n,
                           &zero, ws.gt.p, n) == CUBLAS_STATUS_SUCCESS,
               EQTL_E_CUDA, "Q (w o r) failed");
    U = ws.gt.p;
    u_stride = n;
  }
  float s1, s2;
  output_scales(n, s1, s2);
  ws.tiny_p.alloc(static_cast<size_t>(n_tiny));
  by_sums(ws, n_tiny, p + 2, [&](PairRange pr) {
    const int k = pr.end - pr.first;
    ctx->launches += 2;
    with_p(p, [&](auto pm) {
      lmm_tiny_sums_kernel<decltype(pm)::value><<<static_cast<unsigned>((k + 7) / 8), 256, 0, st>>>(
          g.rows(), g.col.p, n, R.k_pad, g.kept.p, g.mu.p, U, u_stride, R.gt_hi.p, R.gt_lo.p, 1.0 / s1, ws.Xtil.p, p,
          ctx->basis.lambda.p, ws.delta.p, ws.tiny_pairs.p, pr, ws.ref_sums.p);
    });
    lmm_tiny_p_kernel<<<static_cast<unsigned>((k + 63) / 64), 64, 0, st>>>(
        ws.ref_sums.p, ws.tiny_pairs.p, pr, p, ws.ainv.p, ws.rss.p, df, ws.tiny_p.p);
    EQTL_CUDA(cudaGetLastError());
  });
  ws.tiny_p.download(out.data(), out.size(), st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  return out;
}

// Which form of the exact-operand scan (p <= 2, dense) forms gg and a_k:
// interpolated between node deltas (lmm_lr_prepare) from 256 genes on, where
// the node pass costs less than it saves, otherwise directly. EQTL_LMM_FORM
// = "direct" or "lr" fixes the form for every gene count.
static bool lmm_lr_wanted(int G) {
  const char* f = std::getenv("EQTL_LMM_FORM");
  if (f && std::strcmp(f, "direct") == 0) return false;
  if (f && std::strcmp(f, "lr") == 0) return true;
  return G >= 256;
}

// Interpolated gg and a_k: Chebyshev-Lobatto nodes over the genes' range of
// ln(delta) (5 equal intervals if that keeps each within kLrSpan, else 11;
// kLrNodes nodes each, neighbours sharing their end node: 56 or 122 nodes),
// the node genes' operands (w and Q (w o X~_k) at each node delta, as
// lmm_gene_ops_raw_kernel forms a gene's), the node pass over every kept
// SNP, then both sides of the scan's gg and a_k accumulators (ws.lr_phi /
// lr_plo: SNP side [m][kb]; ws.lr_chi / lr_clo: gene side [G][kb];
// ws.unscale of gg and a_k). Returns false, leaving the direct form, when
// the intervals would be longer than kLrSpan.
template <int P>
static bool lmm_lr_build(eqtl_ctx* ctx, int n, int G, const int* gene_row, float s2) {
  Workspace& ws = ctx->ws;
  const Geno& g = ctx->geno;
  const Rotated& R = ctx->rot;
  cudaStream_t st = ctx->stream;
  constexpr int nops = P + 2;
  const int k_pad = g.k_pad;
  const int64_t m = g.m;
  std::vector<double> d(static_cast<size_t>(G));
  ws.delta.download(d.data(), d.size(), st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  double lo = INFINITY, hi = -INFINITY;
  for (double x : d) {
    const double a = std::log(std::max(x, 1e-300));
    if (std::isfinite(a)) {
      lo = std::min(lo, a);
      hi = std::max(hi, a);
    }
  }
  if (!(lo <= hi)) lo = hi = 0.0;
  if (hi - lo < 1e-6) {
    lo -= 0.5;
    hi += 0.5;
  }
  // as many intervals as one or two 64-column chunks of nodes hold (5 or 11)
  const int nint = static_cast<int>(std::ceil((hi - lo) / kLrSpan)) <= 5 ? 5 : 11;
  const double h = (hi - lo) / nint;
  const int nn = nint * (kLrNodes - 1) + 1;
  // intervals longer than kLrSpan (a delta range beyond REML's 1e-8 .. 1e6)
  // would lose the interpolation's accuracy: the direct form then
  if (nn > kTileM || h > kLrSpan * (1.0 + 1e-12)) return false;
  std::vector<double> na(static_cast<size_t>(nn)), nd(static_cast<size_t>(nn));
  for (int q = 0; q < nint; ++q)
    for (int i = 0; i < kLrNodes; ++i)
      na[static_cast<size_t>(q * (kLrNodes - 1) + i)] =
          lo + h * (q + 0.5 * (1.0 - std::cos(M_PI * i / (kLrNodes - 1))));
  for (int j = 0; j < nn; ++j) nd[static_cast<size_t>(j)] = std::exp(na[static_cast<size_t>(j)]);
  const int kn = nn <= 64 ? 64 : 128, kb = (P + 1) * kn;
  ws.lr_kn = kn;
  ws.lr_kb = kb;
  ws.lr_nodes = nn;
  ws.lr_a.upload(na.data(), na.size(), st);
  ws.lr_delta.upload(nd.data(), nd.size(), st);

  // node genes' operands: a zero residual (u = 0), w o X~_k, Q times them
  const size_t cols = static_cast<size_t>(nn) * (P + 1);
  ws.lr_zero.alloc(static_cast<size_t>(nn) * (n + P));
  ws.lr_zero.zero(st);
  ws.lr_w.alloc(static_cast<size_t>(n) * cols);
  ws.lr_uv.alloc(static_cast<size_t>(n) * cols);
  ++ctx->launches;
  lmm_uv_w_kernel<<<nn, 256, 0, st>>>(ws.lr_zero.p, ws.Xtil.p, ctx->basis.lambda.p, ws.lr_delta.p,
                                      ws.lr_zero.p + static_cast<size_t>(nn) * n, n, P, nn, ws.lr_w.p);
  EQTL_CUDA(cudaGetLastError());
  const double one = 1.0, zero = 0.0;
  EQTL_CHECK(cublasDgemm(blas_of(ctx), CUBLAS_OP_N, CUBLAS_OP_N, n, static_cast<int>(cols), n, &one,
                         ctx->basis.Q.p, n, ws.lr_w.p, n, &zero, ws.lr_uv.p, n) == CUBLAS_STATUS_SUCCESS,
             EQTL_E_CUDA, "Q (w o X~) at the node deltas failed");
  ctx->launches += 1;
  __half* nptr[2 * nops];
  for (int k = 0; k < nops; ++k) {
    ws.lr_ops_hi[k].alloc(static_cast<size_t>(nn) * k_pad);
    ws.lr_ops_lo[k].alloc(static_cast<size_t>(nn) * k_pad);
    nptr[k] = ws.lr_ops_hi[k].p;
    nptr[nops + k] = ws.lr_ops_lo[k].p;
  }
  ws.lr_ops_ptr.upload(nptr, 2 * nops, st);
  ws.lr_unscale.alloc(static_cast<size_t>(nn) * nops);
  ++ctx->launches;
  lmm_gene_ops_raw_kernel<<<nn, 256, 0, st>>>(ws.lr_uv.p, ctx->basis.lambda.p, ws.lr_delta.p, n, P, nn, nullptr, k_pad,
                                              s2, ws.lr_ops_ptr.p, ws.lr_ops_ptr.p + nops, ws.lr_unscale.p);
  EQTL_CUDA(cudaGetLastError());

  // node pass: accumulators [gg, a_0 ..] against Gt^2 and the raw operand
  ws.lr_val.alloc(static_cast<size_t>(m) * kb);
  ws.lr_colmax.alloc(static_cast<size_t>(kb));
  ws.lr_colmax.zero(st);
  if (m > 0) {
    LmmNodeEpiParams<P> ep{};
    ep.n_nodes = nn;
    ep.m = m;
    ep.kn = kn;
    ep.kb = kb;
    ep.unscale = ws.lr_unscale.p;
    ep.snp_alpha = R.alpha.p;
    ep.val = ws.lr_val.p;
    ep.colmax = ws.lr_colmax.p;
    const __half* ah[P + 1];
    const __half* al[P + 1];
    int bsel[P + 1], prod[P + 1];
    ah[0] = ws.lr_ops_hi[P + 1].p;
    al[0] = ws.lr_ops_lo[P + 1].p;
    bsel[0] = 1;
    prod[0] = 7;
    for (int k = 0; k < P; ++k) {
      ah[1 + k] = ws.lr_ops_hi[1 + k].p;
      al[1 + k] = ws.lr_ops_lo[1 + k].p;
      bsel[1 + k] = 0;
      prod[1 + k] = 5;
    }
    const __half* bh[2] = {R.raw.p, R.gt2_hi.p};
    const __half* bl[2] = {R.raw.p, R.gt2_lo.p};
    launch_tile_n<128, P + 1>(ctx, false, ep, ah, al, nn, bh, bl, m, k_pad, bsel, prod);
  }
  ws.lr_sigma.alloc(static_cast<size_t>(kb));
  ++ctx->launches;
  lr_sigma_kernel<<<(kb + 255) / 256, 256, 0, st>>>(ws.lr_colmax.p, kb, ws.lr_sigma.p);
  EQTL_CUDA(cudaGetLastError());
  ws.lr_phi.alloc(std::max<size_t>(1, static_cast<size_t>(m) * kb));
  ws.lr_plo.alloc(std::max<size_t>(1, static_cast<size_t>(m) * kb));
  if (m > 0) {
    ++ctx->launches;
    lr_split_kernel<<<4 * sm_count(ctx), 256, 0, st>>>(ws.lr_val.p, m * kb, kb, ws.lr_sigma.p, ws.lr_phi.p,
                                                       ws.lr_plo.p);
    EQTL_CUDA(cudaGetLastError());
  }
  // genes' coefficients (rows zero outside each gene's nodes)
  ws.lr_chi.alloc(static_cast<size_t>(G) * kb);
  ws.lr_clo.alloc(static_cast<size_t>(G) * kb);
  ws.lr_chi.zero(st);
  ws.lr_clo.zero(st);
  ++ctx->launches;
  lr_coef_kernel<<<(G + 127) / 128, 128, 0, st>>>(ws.delta.p, G, ws.lr_a.p, lo, h, nint, ws.lr_sigma.p, kn, kb, P,
                                                  gene_row, ws.lr_chi.p, ws.lr_clo.p, ws.unscale.p);
  EQTL_CUDA(cudaGetLastError());
  return true;
}

// lmm_lr_build, or the direct form when its tables do not fit in device
// memory beside the scan's operands (their large buffers are given back).
template <int P>
static bool lmm_lr_prepare(eqtl_ctx* ctx, int n, int G, const int* gene_row, float s2) {
  try {
    return lmm_lr_build<P>(ctx, n, G, gene_row, s2);
  } catch (const Error& e) {
    if (e.code != EQTL_E_NOMEM) throw;
    EQTL_CUDA(cudaStreamSynchronize(ctx->stream));
    (void)cudaGetLastError();  // the failed allocation's error, so later launch checks do not see it
    Workspace& ws = ctx->ws;
    ws.lr_val.release();
    ws.lr_phi.release();
    ws.lr_plo.release();
    ws.lr_chi.release();
    ws.lr_clo.release();
    ws.lr_nodes = 0;
    return false;
  }
}

// The scan with interpolated gg and a_k, in LmmEpi's accumulator order: gg
// and a_k read their kind's node columns of both interpolated operands
// (K chunks [kind c, (kind + 1) c), c = kn / 64), NUM reads u hi + lo
// against the exact raw operand over all of K. ah / al: the gene-ops order
// [NUM, a_0 .., gg] (only NUM's u is read).
template <int P>
static void lmm_launch_lr(eqtl_ctx* ctx, const LmmLrEpiParams<P>& ep, const __half* const* ah,
                          const __half* const* al, int G, const Rotated& R) {
  Workspace& ws = ctx->ws;
  const int kb = ws.lr_kb, c = ws.lr_kn / kChunkK;
  const __half* oh[P + 2];
  const __half* ol[P + 2];
  int bsel[P + 2], prod[P + 2];
  TileK tk;
  for (int j = 0; j < P + 2; ++j) {
    const int op = lmm_acc_op(P, j, true);
    if (op == 0) {
      oh[j] = ah[0];
      ol[j] = al[0];
      bsel[j] = 0;
      prod[j] = 5;
      continue;
    }
    const int kind = op == P + 1 ? 0 : op;  // lr_coef_kernel's order: gg, a_0 ..
    oh[j] = ws.lr_chi.p;
    ol[j] = ws.lr_clo.p;
    bsel[j] = 1;
    prod[j] = 7;
    tk.beg[j] = kind * c;
    tk.end[j] = (kind + 1) * c;
    tk.k_a[j] = kb;
  }
  tk.k_b[1] = kb;
  const __half* bh[2] = {R.raw.p, ws.lr_phi.p};
  const __half* bl[2] = {R.raw.p, ws.lr_plo.p};
  launch_tile_n<128, P + 2>(ctx, false, ep, oh, ol, G, bh, bl, R.m, R.k_pad, bsel, prod, nullptr, 0, 1, P + 2, 0,
                            &tk);
}

// The grouped scan (p >= 3): ops = the gene-side hi operands [NUM, gg, a~_0 ..],
// then their lo parts; bh / bl = [Gt, Gt^2]. Dense scans run on SM pairs.
template <class EP>
static void launch_grouped(eqtl_ctx* ctx, bool bf16, const EP& ep, const __half* const* ops, int nops, int G,
                           const __half* const* bh, const __half* const* bl, int64_t m, int k_pad, const int2* tiles,
                           int n_tiles) {
  using E = typename EpiOf<EP>::type;
  std::vector<const __half*> ah(static_cast<size_t>(nops)), al(static_cast<size_t>(nops));
  std::vector<int> bsel(static_cast<size_t>(nops)), prod(static_cast<size_t>(nops), 7);
  for (int j = 0; j < nops; ++j) {
    const int op = j == nops - 1 ? 0 : j + 1;  // tile order [gg, a~_0 .., NUM]
    ah[static_cast<size_t>(j)] = ops[op];
    al[static_cast<size_t>(j)] = ops[nops + op];
    bsel[static_cast<size_t>(j)] = op == 1 ? 1 : 0;  // gg reads the squares
  }
  if (!bf16 && !tiles && tile_pairs(G))
    launch_tile_n<E::kTileN, E::kGroup, EP, dev::kBLoStage, 2>(ctx, false, ep, ah.data(), al.data(), G, bh, bl, m,
                                                               k_pad, bsel.data(), prod.data(), nullptr, 0, 1, nops);
  else
    launch_tile_n<E::kTileN, E::kGroup>(ctx, bf16, ep, ah.data(), al.data(), G, bh, bl, m, k_pad, bsel.data(),
                                        prod.data(), tiles, n_tiles, 1, nops);
}

// Subset gate of every kept SNP on the analysis samples into ws.ok.
static void lmm_gate(eqtl_ctx* ctx) {
  Geno& g = ctx->geno;
  DevBuf<uint8_t>& ok = ctx->ws.ok;
  const int64_t m = g.m;
  ok.alloc(static_cast<size_t>(((m + 255) / 256 + 1) * 256));  // the epilogue reads 16 flags per chunk, up to the last tile's end
  EQTL_CUDA(cudaMemsetAsync(ok.p, 0, ok.n, ctx->stream));
  if (m > 0) {
    ++ctx->launches;
    snp_gate_kernel<<<static_cast<unsigned>((m + 255) / 256), 256, 0, ctx->stream>>>(g.kept.p, m, g.n, g.mu.p,
                                                                                     g.gate_nmiss(), g.gate_s1(), g.gate_s2(), ok.p);
    EQTL_CUDA(cudaGetLastError());
  }
}

static void scan_trans_lmm_impl(eqtl_ctx* ctx, const eqtl_scan_params* prm, const double* Y, const double* X,
                                double* delta_out, eqtl_gene_result* genes, PairList& pairs, PairList& cands, bool simt) {
  Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  const int n = prm->n, G = prm->n_genes, p = prm->p;
  EQTL_CHECK(g.m_all > 0, EQTL_E_STATE, "scan_trans_lmm: no genotypes loaded");
  EQTL_CHECK(n == g.n, EQTL_E_ARG, "scan_trans_lmm: n differs from the loaded genotypes");
  EQTL_CHECK(G > 0, EQTL_E_ARG, "scan_trans_lmm: no genes");
  EQTL_CHECK(g.m < (int64_t(1) << 30), EQTL_E_UNSUPPORTED, "scan_trans_lmm: more than 2^30 kept SNPs");
  EQTL_CHECK(p >= 1 && p <= kMaxPLmm, EQTL_E_UNSUPPORTED,
             "the LMM scan handles 1 to 32 covariate columns (intercept included)");
  EQTL_CHECK(!(simt && p > 2), EQTL_E_UNSUPPORTED, "the FP32 CUDA-core comparator covers 1 or 2 covariate columns");
  const bool grouped = p > 2;  // accumulators run in groups of two (LmmGroupEpi)
  cudaStream_t st = ctx->stream;
  const double df = static_cast<double>(n - p - 1);
  const PhenoDev& ph = resolve_pheno(ctx, prm, Y, X);
  lmm_rotate(ctx);
  // p <= 2 on the tensor cores: NUM and a_k from the exact unrotated SNP
  // operand when every kept SNP fits it (2-bit rows, FP16 operands)
  const bool raw = !grouped && !simt && ctx->precision == EQTL_PREC_SPLIT_F16 && geno_raw_operand(ctx);
  std::unique_ptr<StageScope> prep_timer(new StageScope(ctx, EQTL_STAGE_PREP));
  lmm_prep(ctx, ph, prm->y_rotated != 0);

  // gene-side operands
  const GeneOrder go = gene_order(ctx, prm);
  const int k_pad = g.k_pad;
  const int nops = p + 2;
  float s1, s2;
  output_scales(n, s1, s2);
  std::vector<__half*> oph(2 * nops);
  for (int k = 0; k < nops; ++k) {
    ws.ops_hi[k].alloc(static_cast<size_t>(G) * k_pad);
    ws.ops_lo[k].alloc(static_cast<size_t>(G) * k_pad);
    oph[k] = ws.ops_hi[k].p;
    oph[nops + k] = ws.ops_lo[k].p;
  }
  ws.ops_ptr.upload(oph.data(), oph.size(), st);
  DevBuf<float>& unscale = ws.unscale;
  unscale.alloc(static_cast<size_t>(G) * nops);
  ++ctx->launches;
  if (raw) {
    // u = Q (w o r~) and v_k = Q (w o X~_k) in FP64, then their FP16 hi/lo
    const size_t cols = static_cast<size_t>(G) * (p + 1);
    ws.lmm_w.alloc(static_cast<size_t>(n) * cols);
    ws.lmm_uv.alloc(static_cast<size_t>(n) * cols);
    lmm_uv_w_kernel<<<G, 256, 0, st>>>(ws.Ytil.p, ws.Xtil.p, ctx->basis.lambda.p, ws.delta.p, ws.chi0.p, n, p, G,
                                       ws.lmm_w.p);
    EQTL_CUDA(cudaGetLastError());
    const double one = 1.0, zero = 0.0;
    EQTL_CHECK(cublasDgemm(blas_of(ctx), CUBLAS_OP_N, CUBLAS_OP_N, n, static_cast<int>(cols), n, &one,
                           ctx->basis.Q.p, n, ws.lmm_w.p, n, &zero, ws.lmm_uv.p, n) == CUBLAS_STATUS_SUCCESS,
               EQTL_E_CUDA, "Q (w o [r~, X~]) failed");
    ctx->launches += 1;
    lmm_gene_ops_raw_kernel<<<G, 256, 0, st>>>(ws.lmm_uv.p, ctx->basis.lambda.p, ws.delta.p, n, p, G, go.row, k_pad,
                                               s2, ws.ops_ptr.p, ws.ops_ptr.p + nops, unscale.p);
  } else if (grouped) {
    auto run = [&](auto pm) {
      lmm_gene_ops_orth_kernel<decltype(pm)::value><<<G, 256, 0, st>>>(
          ws.Ytil.p, ws.Xtil.p, ctx->basis.lambda.p, ws.delta.p, ws.chi0.p, ws.ainv.p, n, p, G, go.row, k_pad, s1, s2,
          ws.ops_ptr.p, ws.ops_ptr.p + nops, unscale.p);
    };
    if (p <= 4) run(std::integral_constant<int, 4>{});
    else if (p <= 8) run(std::integral_constant<int, 8>{});
    else if (p <= 16) run(std::integral_constant<int, 16>{});
    else run(std::integral_constant<int, kMaxPLmm>{});
  } else {
    lmm_gene_ops_kernel<<<G, 256, 0, st>>>(ws.Ytil.p, ws.Xtil.p, ctx->basis.lambda.p, ws.delta.p, ws.chi0.p, n, p, G,
                                           go.row, k_pad, s1, s2, ws.ops_ptr.p, ws.ops_ptr.p + nops, unscale.p);
  }
  EQTL_CUDA(cudaGetLastError());
  // dense scans with the exact operand: gg and a_k interpolated between node
  // deltas when that pays (lmm_lr_wanted)
  bool lr = false;
  ws.lr_nodes = 0;
  if (raw && prm->exclude_cis != 2 && lmm_lr_wanted(G))
    lr = p == 1 ? lmm_lr_prepare<1>(ctx, n, G, go.row, s2) : lmm_lr_prepare<2>(ctx, n, G, go.row, s2);
  if (simt) {
    // the FP32 form's gene-side operands, in the tile's accumulator order
    // [gg, a_0 .. a_{p-1}, NUM] (the gene-ops order is [NUM, a.., gg])
    for (int j = 0; j < nops; ++j) {
      const int op = j == 0 ? nops - 1 : (j == nops - 1 ? 0 : j);
      ws.ops32[j].alloc(static_cast<size_t>(G) * k_pad);
      ++ctx->launches;
      sum_split_kernel<<<1184, 256, 0, st>>>(ws.ops_hi[op].p, ws.ops_lo[op].p, static_cast<int64_t>(G) * k_pad,
                                             ws.ops32[j].p);
    }
    EQTL_CUDA(cudaGetLastError());
  }

  const int64_t m = g.m;
  lmm_gate(ctx);
  DevBuf<uint8_t>& ok = ws.ok;
  const Windows win = upload_windows(ctx, prm, m, prm->exclude_cis == 2 ? kWinInclude : prm->exclude_cis ? kWinExclude : kWinNone);
  double t_cand = t_critical(prm->pthr, df);
  if (prm->perm_thr > 0) t_cand = std::min(t_cand, t_critical(prm->perm_thr, df));
  const TTable tt = device_ttable(ctx, df);
  prep_timer.reset();
  ScanOutputs so(ctx, G, m, expected_candidates(prm, m));
  const int2* tiles = nullptr;  // cis: banded tile list (NT of the kernel that runs)
  int n_tiles = 0;
  if (!simt) cis_tile_list(ctx, win, G, go, m, grouped ? LmmGroupEpi::kTileN : 128, tiles, n_tiles);
  std::unique_ptr<StageScope> scan_timer(new StageScope(ctx, EQTL_STAGE_SCAN));
  if (m > 0 && grouped) {
    Rotated& Rt = ctx->rot;
    LmmGroupEpiParams ep{};
    ep.G = G;
    ep.order = go.gene;
    ep.m = m;
    ep.n_acc = nops;
    ep.unscale = unscale.p;
    ep.rss_null = ws.rss.p;
    ep.snp_ok = ok.p;
    ep.win = win;
    ep.df = static_cast<float>(df);
    ep.t_cand = static_cast<float>(t_cand * (1.0 - 1e-3));
    ep.tt = tt;
    const __half* bh[2] = {Rt.gt_hi.p, Rt.gt2_hi.p};
    const __half* bl[2] = {Rt.gt_lo.p, Rt.gt2_lo.p};
    const bool bf16 = ctx->precision == EQTL_PREC_SPLIT_BF16;
    std::vector<const __half*> opb(2 * static_cast<size_t>(nops));
    if (bf16) {
      // split-BF16: both sides re-split into BF16 hi + lo
      gene_ops_bf16(ctx, oph.data(), oph.data() + nops, nops, G, Rt.k_pad, opb.data());
      rot_bf16(ctx, Rt);
      bh[0] = Rt.bgt_hi.p;
      bh[1] = Rt.bgt2_hi.p;
      bl[0] = Rt.bgt_lo.p;
      bl[1] = Rt.bgt2_lo.p;
    }
    const __half* const* ops = bf16 ? opb.data() : oph.data();
    so.run([&](GeneOut out) {
      ep.out = out;
      launch_grouped(ctx, bf16, ep, ops, nops, G, bh, bl, Rt.m, Rt.k_pad, tiles, n_tiles);
    });
  } else if (m > 0) {
    const __half* ah[4] = {oph[0], oph[1], oph[2], nops > 3 ? oph[3] : oph[2]};
    const __half* al[4] = {oph[nops + 0], oph[nops + 1], oph[nops + 2], nops > 3 ? oph[nops + 3] : oph[nops + 2]};
    auto fill = [&](auto& ep) {
      ep.G = G;
      ep.order = go.gene;
      ep.m = m;
      ep.unscale = unscale.p;
      ep.ainv = ws.ainv.p;
      ep.rss_null = ws.rss.p;
      ep.snp_ok = ok.p;
      ep.win = win;
      ep.df = static_cast<float>(df);
      ep.t_cand = static_cast<float>(t_cand * (1.0 - 1e-3));
      ep.tt = tt;
    };
    auto run = [&](auto ep, auto pc) {
      constexpr int P = decltype(pc)::value;
      fill(ep);
      ep.snp_alpha = ctx->rot.alpha.p;
      so.run([&](GeneOut out) {
        ep.out = out;
        if constexpr (std::is_same_v<std::decay_t<decltype(ep)>, LmmLrEpiParams<P>>) lmm_launch_lr<P>(ctx, ep, ah, al, G, ctx->rot);
        else lmm_launch<P>(ctx, ep, ah, al, G, simt, tiles, n_tiles, ctx->rot);
      });
    };
    using P1 = std::integral_constant<int, 1>;
    using P2 = std::integral_constant<int, 2>;
    if (lr && p == 1) run(LmmLrEpiParams<1>{}, P1{});
    else if (lr) run(LmmLrEpiParams<2>{}, P2{});
    else if (raw && p == 1) run(LmmRawEpiParams<1>{}, P1{});
    else if (raw) run(LmmRawEpiParams<2>{}, P2{});
    else if (p == 1) run(LmmEpiParams<1>{}, P1{});
    else run(LmmEpiParams<2>{}, P2{});
  }
  scan_timer.reset();
  HostTrace tr("scan_trans_lmm");
  so.collect(true);
  tr.mark("collect (waits for the scan)");

  // ---- FP64 refinement: rotate raw dosages of the SNPs involved
  StageScope refine_timer(ctx, EQTL_STAGE_REFINE);
  if (delta_out) {
    ws.delta.download(delta_out, G, st);
    EQTL_CUDA(cudaStreamSynchronize(st));
  }
  lmm_refine_pairs(ctx, p, df, so.n_todo);
  tr.mark("refine pairs");
  const std::vector<double> tiny_p = raw ? lmm_tiny_p(ctx, p, df, so.n_tiny, ws.lmm_uv.p, static_cast<int64_t>(p + 1) * n)
                                         : lmm_tiny_p(ctx, p, df, so.n_tiny);
  std::vector<int2> tiny(static_cast<size_t>(so.n_tiny));
  ws.tiny_pairs.download(tiny.data(), tiny.size(), st);
  tr.mark("tiny-|t| pairs");
  so.finish(prm, genes, pairs, cands);
  tr.mark("finish");
  add_acat_terms(genes, tiny, tiny_p);
  tr.mark("tiny ACAT terms");
  if (tr.on)
    std::fprintf(stderr, "[eqtl trace] scan_trans_lmm counts: candidates %d deferred %d tiny %d\n", so.n_todo,
                 so.n_deferred, so.n_tiny);
}

void scan_trans_lmm(eqtl_ctx* ctx, const eqtl_scan_params* prm, const double* Y, const double* X, double* delta_out,
                    eqtl_gene_result* genes, PairList& pairs, PairList& cands) {
  scan_trans_lmm_impl(ctx, prm, Y, X, delta_out, genes, pairs, cands, false);
}

void scan_trans_lmm_simt(eqtl_ctx* ctx, const eqtl_scan_params* prm, const double* Y, const double* X,
                         double* delta_out, eqtl_gene_result* genes, PairList& pairs, PairList& cands) {
  scan_trans_lmm_impl(ctx, prm, Y, X, delta_out, genes, pairs, cands, true);
}

// FP64 tests of explicit (column of Y, kept SNP) pairs with the resident
// eigenbasis: the full null fit per column (Q'Y, REML delta, GLS), then the
// refinement arithmetic of the scan; a SNP that fails the subset gate gets
// p = NaN (it is never tested in the reference).
void test_pairs_lmm(eqtl_ctx* ctx, const eqtl_scan_params* prm, const double* Y, const double* X,
                    const std::vector<int2>& todo, eqtl_pair* out, double* delta_out) {
  Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  EQTL_CHECK(g.m_all > 0, EQTL_E_STATE, "test_pairs: no genotypes loaded");
  const int n = prm->n, G = prm->n_genes, p = prm->p;
  EQTL_CHECK(n == g.n, EQTL_E_ARG, "test_pairs: n differs from the loaded genotypes");
  EQTL_CHECK(G > 0, EQTL_E_ARG, "test_pairs: no columns");
  for (const int2& q : todo)
    EQTL_CHECK(q.x >= 0 && q.x < G && q.y >= 0 && q.y < g.m, EQTL_E_ARG, "test_pairs: pair index out of range");
  const double df = static_cast<double>(n - p - 1);
  const PhenoDev& ph = resolve_pheno(ctx, prm, Y, X);
  lmm_prep(ctx, ph, prm->y_rotated != 0);
  lmm_gate(ctx);
  std::vector<uint8_t> ok(static_cast<size_t>(g.m));
  ws.ok.download(ok.data(), static_cast<size_t>(g.m), ctx->stream);
  ws.ref_pairs.upload(todo.data(), todo.size(), ctx->stream);
  lmm_refine_pairs(ctx, p, df, static_cast<int>(todo.size()));
  ws.refined.download(out, todo.size(), ctx->stream);
  EQTL_CUDA(cudaStreamSynchronize(ctx->stream));
  for (size_t i = 0; i < todo.size(); ++i)
    if (!ok[todo[i].y]) out[i].p = std::numeric_limits<double>::quiet_NaN();
  if (delta_out) {
    ws.delta.download(delta_out, G, ctx->stream);
    EQTL_CUDA(cudaStreamSynchronize(ctx->stream));
  }
}


// ================================================================ NB GLM
// The NB-GLM score test (src/model_glm.cpp:13-132) on the LMM scan's
// machinery: the null fit of every gene on the device (glm_null_kernel), the
// gene-side operands w, w o x_k (or w o (X U)_k, U U' = (X'WX)^-1, for
// p > 2) and r against the unrotated centred dosages gc and gc^2, the
// score-test epilogues (LmmEpi<P, true>, GlmGroupEpi), and the FP64
// refinement of every candidate from the exact dosages (glm_pair_sums_kernel).
namespace dev {

constexpr int kGlmThreads = 256;

// Null NB2 fit of one gene per block (nb_irls + prep_glm_nb, src/model_glm.cpp:
// 28-96): from beta = 0, mu = max(y, 0.1), phi = 1, IRLS at fixed phi (at most
// 50 rounds, until max |beta change| < 1e-6; w = m^2 / (m + phi m^2),
// z = log m + (y - m) / m, m = max(mu, 1e-8)), then phi by moments
// (sum ((y - m)^2 - m) / m^2 / max(1, n - p), at least 1e-8), until phi moves
// by less than 1e-6 max(1, phi) (at most 10 rounds). The sums of X'WX and X'Wz
// are warp dot products over the samples (warp w takes items w, w + 8, ...);
// thread 0 factorises and solves. Outputs per gene: W = m / (1 + phi m),
// R = (y - mu) / (1 + phi mu), (X'WX)^-1, phi, sum R, ok (every X'WX
// factorised) and counts (every y a non-negative integer within 1e-8).
// MU and R double as the fit's mu and z.
__global__ void __launch_bounds__(kGlmThreads)
    glm_null_kernel(const double* __restrict__ Y, const double* __restrict__ X, int n, int p, int G, double* MU,
                    double* W, double* R, double* phi_out, double* ainv_out, double* rsum_out, uint8_t* ok_out,
                    uint8_t* counts_out) {
  const int g = blockIdx.x;
  if (g >= G) return;
  __shared__ double A[kMaxPLmm * kMaxPLmm];
  __shared__ double rhs[kMaxPLmm], beta[kMaxPLmm], sol[kMaxPLmm];
  __shared__ double red[kGlmThreads / 32];
  __shared__ double s_phi, s_diff;
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nw = kGlmThreads / 32;
  const double* y = Y + static_cast<int64_t>(g) * n;
  double* mu = MU + static_cast<int64_t>(g) * n;
  double* w = W + static_cast<int64_t>(g) * n;
  double* z = R + static_cast<int64_t>(g) * n;
  auto block_sum = [&](double v) -> double {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();  // red[] of the previous sum has been read
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0;
    for (int k = 0; k < nw; ++k) t += red[k];
    return t;
  };
  // X'WX (lower triangle, items 0 .. p(p+1)/2 - 1) and, with rhs, X'Wz
  const int n_tri = p * (p + 1) / 2;
  auto weighted_sums = [&](bool with_rhs) {
    const int items = n_tri + (with_rhs ? p : 0);
    for (int item = warp; item < items; item += nw) {
      int a = 0, b = 0;
      const bool is_rhs = item >= n_tri;
      if (is_rhs) {
        a = item - n_tri;
      } else {
        while ((a + 1) * (a + 2) / 2 <= item) ++a;
        b = item - a * (a + 1) / 2;
      }
      const double* xa = X + static_cast<int64_t>(a) * n;
      const double* xb = X + static_cast<int64_t>(b) * n;
      double acc = 0;
      for (int i = lane; i < n; i += 32) acc += xa[i] * w[i] * (is_rhs ? z[i] : xb[i]);
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) {
        if (is_rhs) {
          rhs[a] = acc;
        } else {
          A[a * p + b] = acc;
          A[b * p + a] = acc;
        }
      }
    }
  };
  // thread 0: lower Cholesky factor of A in place; false if A is not
  // positive definite
  auto cholesky = [&]() -> bool {
    for (int j = 0; j < p; ++j) {
      double d = A[j * p + j];
      for (int k = 0; k < j; ++k) d -= A[j * p + k] * A[j * p + k];
      if (!(d > 0)) return false;
      d = sqrt(d);
      A[j * p + j] = d;
      for (int i = j + 1; i < p; ++i) {
        double v = A[i * p + j];
        for (int k = 0; k < j; ++k) v -= A[i * p + k] * A[j * p + k];
        A[i * p + j] = v / d;
      }
    }
    return true;
  };
  // thread 0: sol = (L L')^-1 v with the factor in A's lower triangle
  auto solve = [&](const double* v) {
    for (int i = 0; i < p; ++i) {
      double t = v[i];
      for (int k = 0; k < i; ++k) t -= A[i * p + k] * sol[k];
      sol[i] = t / A[i * p + i];
    }
    for (int i = p - 1; i >= 0; --i) {
      double t = sol[i];
      for (int k = i + 1; k < p; ++k) t -= A[k * p + i] * sol[k];
      sol[i] = t / A[i * p + i];
    }
  };

  double bad = 0;
  for (int i = tid; i < n; i += kGlmThreads) {
    const double v = y[i];
    if (isfinite(v) && (v < 0 || fabs(v - floor(v)) > 1e-8)) bad = 1;
    mu[i] = fmax(v, 0.1);
  }
  const double n_bad = block_sum(bad);
  if (tid < p) beta[tid] = 0.0;
  if (tid == 0) {
    s_phi = 1.0;
    s_fail = 0;
  }
  __syncthreads();
  const int df = n - p > 1 ? n - p : 1;
  for (int outer = 0; outer < 10; ++outer) {
    for (int it = 0; it < 50; ++it) {
      const double phi = s_phi;
      for (int i = tid; i < n; i += kGlmThreads) {
        const double m = fmax(mu[i], 1e-8);
        const double var = m + phi * m * m;
        w[i] = (m * m) / fmax(var, 1e-12);
        z[i] = log(m) + (y[i] - m) / m;
      }
      __syncthreads();
      weighted_sums(true);
      __syncthreads();
      if (tid == 0) {
        if (!cholesky()) {
          s_fail = 1;
        } else {
          solve(rhs);
          double diff = 0;
          for (int k = 0; k < p; ++k) {
            diff = fmax(diff, fabs(sol[k] - beta[k]));
            beta[k] = sol[k];
          }
          s_diff = diff;
        }
      }
      __syncthreads();
      if (s_fail) break;
      for (int i = tid; i < n; i += kGlmThreads) {
        double e = 0;
        for (int k = 0; k < p; ++k) e += X[static_cast<int64_t>(k) * n + i] * beta[k];
        mu[i] = exp(e);
      }
      __syncthreads();
      if (s_diff < 1e-6) break;
    }
    if (s_fail) break;
    double part = 0;
    for (int i = tid; i < n; i += kGlmThreads) {
      const double m = fmax(mu[i], 1e-8);
      part += ((y[i] - m) * (y[i] - m) - m) / (m * m);
    }
    const double phi_new = fmax(1e-8, block_sum(part) / df);
    const double phi = s_phi;
    __syncthreads();
    if (tid == 0) s_phi = phi_new;
    __syncthreads();
    if (fabs(phi_new - phi) < 1e-6 * fmax(1.0, phi)) break;
  }
  // the fitted null's weights, residuals and (X'WX)^-1
  const double phi = s_phi;
  double rpart = 0;
  for (int i = tid; i < n; i += kGlmThreads) {
    const double m = fmax(mu[i], 1e-8);
    w[i] = m / (1.0 + phi * m);
    const double r = (y[i] - mu[i]) / (1.0 + phi * mu[i]);
    z[i] = r;
    rpart += r;
  }
  const double rs = block_sum(rpart);
  weighted_sums(false);
  __syncthreads();
  if (tid == 0) {
    const bool fact = cholesky();
    double* ai = ainv_out + static_cast<int64_t>(g) * p * p;
    for (int c = 0; c < p; ++c) {
      for (int k = 0; k < p; ++k) rhs[k] = k == c ? 1.0 : 0.0;
      if (fact) solve(rhs);
      for (int k = 0; k < p; ++k) ai[k * p + c] = fact ? sol[k] : 0.0;
    }
    phi_out[g] = phi;
    rsum_out[g] = rs;
    ok_out[g] = (!s_fail && fact) ? 1 : 0;
    counts_out[g] = n_bad == 0 ? 1 : 0;
  }
}

// Gene-side operands of the GLM scan in the LMM kernels' layout (see
// lmm_gene_ops_kernel / lmm_gene_ops_orth_kernel): order [NUM, a_0 ..
// a_{p-1}, gg] = [r, w x_k, w] for p <= 2, [NUM, gg, a~_0 ..] = [r, w,
// w (X U)_k] for the grouped scan, U the lower Cholesky factor of
// (X'WX)^-1; each scaled to a power of two and split into FP16 hi + lo.
__global__ void glm_gene_ops_kernel(const double* __restrict__ W, const double* __restrict__ Rr,
                                    const double* __restrict__ X, const double* __restrict__ ainv, int n, int p, int G,
                                    const int* __restrict__ gene_row, int k_pad, float s1, float s2, int grouped,
                                    __half* const* hi, __half* const* lo, float* unscale) {
  const int g = blockIdx.x;
  if (g >= G) return;
  const int64_t row = gene_row ? gene_row[g] : g;  // operand row
  const int nops = p + 2;
  __shared__ double mx[kMaxPLmm + 2][8];
  __shared__ double sc[kMaxPLmm + 2];
  __shared__ double U[kMaxPLmm * kMaxPLmm];
  if (grouped && threadIdx.x == 0) {
    const double* A = ainv + static_cast<int64_t>(g) * p * p;
    for (int j = 0; j < p; ++j) {
      double d = A[j * p + j];
      for (int k = 0; k < j; ++k) d -= U[j * p + k] * U[j * p + k];
      d = d > 0 ? sqrt(d) : 0.0;
      U[j * p + j] = d;
      for (int i = j + 1; i < p; ++i) {
        double v = A[i * p + j];
        for (int k = 0; k < j; ++k) v -= U[i * p + k] * U[j * p + k];
        U[i * p + j] = d > 0 ? v / d : 0.0;
      }
      for (int i = 0; i < j; ++i) U[i * p + j] = 0.0;
    }
  }
  __syncthreads();
  const double* wg = W + static_cast<int64_t>(g) * n;
  const double* rg = Rr + static_cast<int64_t>(g) * n;
  const int gg_op = grouped ? 1 : nops - 1;
  auto value = [&](int op, int i) -> double {
    if (i >= n) return 0.0;
    if (op == 0) return rg[i];
    if (op == gg_op) return wg[i];
    if (!grouped) return wg[i] * X[static_cast<int64_t>(op - 1) * n + i];
    const int k = op - 2;
    double v = 0;
    for (int l = k; l < p; ++l) v += X[static_cast<int64_t>(l) * n + i] * U[l * p + k];
    return wg[i] * v;
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int op = 0; op < nops; ++op) {
    double m = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fabs(value(op, i)));
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) mx[op][warp] = m;
  }
  __syncthreads();
  if (threadIdx.x < nops) {
    double m = 0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) m = fmax(m, mx[threadIdx.x][w]);
    int e = 0;
    if (m > 0) e = 10 - static_cast<int>(floor(log2(m)));
    sc[threadIdx.x] = ldexp(1.0, e);
    const double side = static_cast<int>(threadIdx.x) == gg_op ? s2 : s1;
    unscale[static_cast<int64_t>(g) * nops + threadIdx.x] = static_cast<float>(1.0 / (ldexp(1.0, e) * side));
  }
  __syncthreads();
  for (int op = 0; op < nops; ++op) {
    const double sv = sc[op];
    for (int i = threadIdx.x; i < k_pad; i += blockDim.x) {
      const double v = value(op, i) * sv;
      const __half h = __double2half(v);
      hi[op][row * k_pad + i] = h;
      lo[op][row * k_pad + i] = __double2half(v - static_cast<double>(__half2float(h)));
    }
  }
}

// SNP-side operands of the GLM scan: gc * s1 and gc^2 * s2 from the centred
// dosage operand (gc_hi + gc_lo = (dosage - mean) * inv_gc^-1), FP16 hi + lo.
__global__ void glm_snp_ops_kernel(const __half* __restrict__ gc_hi, const __half* __restrict__ gc_lo, int64_t elems,
                                   double inv_gc, float s1, float s2, __half* gh, __half* gl, __half* g2h,
                                   __half* g2l) {
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < elems;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double v = (static_cast<double>(__half2float(gc_hi[e])) + static_cast<double>(__half2float(gc_lo[e]))) *
                     inv_gc;
    const double a = v * s1, b = v * v * s2;
    const __half ah = __double2half(a), bh = __double2half(b);
    gh[e] = ah;
    gl[e] = __double2half(a - static_cast<double>(__half2float(ah)));
    g2h[e] = bh;
    g2l[e] = __double2half(b - static_cast<double>(__half2float(bh)));
  }
}

// FP32 imputation mean of every kept SNP (zero past m), and FP32 sum r
__global__ void glm_means_kernel(const int64_t* __restrict__ kept, int64_t m, const double* __restrict__ mu,
                                 int64_t padded, float* mean_f, const double* __restrict__ rsum, int G, float* rsum_f) {
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < padded;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    mean_f[r] = r < m ? static_cast<float>(mu[kept[r]]) : 0.0f;
    if (r < G) rsum_f[r] = static_cast<float>(rsum[r]);
  }
}

// One warp per (gene, kept SNP) pair: the score test in FP64 from the exact
// mean-imputed dosages g, as test_glm_nb computes it: U = g'r, g'Wg,
// X'Wg, and the dosage variance (mean of squares - squared mean).
// Sums [U, g'Wg, sum g, sum g^2, (X'Wg)_k] by a warp per pair, then the statistics by a
// thread per pair, as for the LMM. n = 1000, p = 3, 2e8 tests: 0.35 -> 0.07 ms.
template <int PM>
__global__ void glm_pair_sums_kernel(GenoRows src, const int32_t* __restrict__ col, int n,
                                     const int64_t* __restrict__ kept, const double* __restrict__ mu_imp,
                                     const double* __restrict__ W, const double* __restrict__ Rr,
                                     const double* __restrict__ X, int p, const int2* __restrict__ pairs, PairRange pr,
                                     double* __restrict__ sums) {
  const int lane = threadIdx.x & 31;
  const int wid = pr.first + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wid >= pr.end) return;
  const int g = pairs[wid].x;
  const int64_t s = kept[pairs[wid].y];
  const double mus = mu_imp[s];
  const double* wg = W + static_cast<int64_t>(g) * n;
  const double* rg = Rr + static_cast<int64_t>(g) * n;
  double U = 0, gwg = 0, sd = 0, sd2 = 0, xw[PM];
#pragma unroll
  for (int k = 0; k < PM; ++k) xw[k] = 0;
#pragma unroll(PM <= 4 ? 8 : 2)
  for (int i = lane; i < n; i += 32) {
    double d = src.dosage(s, col[i]);
    if (isnan(d)) d = mus;
    const double wd = wg[i] * d;
    U += d * rg[i];
    gwg += wd * d;
    sd += d;
    sd2 += d * d;
#pragma unroll
    for (int k = 0; k < PM; ++k)
      if (k < p) xw[k] += X[static_cast<int64_t>(k) * n + i] * wd;
  }
  for (int o = 16; o; o >>= 1) {
    U += __shfl_xor_sync(0xffffffffu, U, o);
    gwg += __shfl_xor_sync(0xffffffffu, gwg, o);
    sd += __shfl_xor_sync(0xffffffffu, sd, o);
    sd2 += __shfl_xor_sync(0xffffffffu, sd2, o);
#pragma unroll
    for (int k = 0; k < PM; ++k)
      if (k < p) xw[k] += __shfl_xor_sync(0xffffffffu, xw[k], o);
  }
  if (lane != 0) return;
  double* out = sums + static_cast<int64_t>(wid - pr.first) * (p + 4);
  out[0] = U;
  out[1] = gwg;
  out[2] = sd;
  out[3] = sd2;
#pragma unroll
  for (int k = 0; k < PM; ++k)
    if (k < p) out[4 + k] = xw[k];
}
__global__ void glm_pair_stats_kernel(const double* __restrict__ sums, int n, int p, const double* __restrict__ ainv,
                                      const uint8_t* __restrict__ gene_ok, const int2* __restrict__ pairs, PairRange pr,
                                      eqtl_pair* __restrict__ out) {
  const int wid = pr.first + blockIdx.x * blockDim.x + threadIdx.x;
  if (wid >= pr.end) return;
  const int g = pairs[wid].x;
  const double* s = sums + static_cast<int64_t>(wid - pr.first) * (p + 4);
  const double* xw = s + 4;
  const double* A = ainv + static_cast<int64_t>(g) * p * p;
  double xAx = 0;
  for (int a = 0; a < p; ++a) {
    double t = 0;
    for (int b = 0; b < p; ++b) t += A[a * p + b] * xw[b];
    xAx += xw[a] * t;
  }
  const double mean = s[2] / n;
  eqtl_pair q;
  q.snp = pairs[wid].y;
  q.gene = g;
  q.reserved = 0;
  glm_stats_fp64(s[0], s[1], xAx, s[3] / n - mean * mean, q);
  // a gene whose null fit failed tests nothing (p = NaN, test_glm_nb)
  if (!gene_ok[g]) q.p = CUDART_NAN;
  out[wid] = q;
}

}  // namespace dev

// FP64 statistics of the first n_pairs of ws.ref_pairs into ws.refined.
static void glm_refine_pairs(eqtl_ctx* ctx, int p, int n_pairs) {
  Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  if (n_pairs == 0) return;
  ws.refined.alloc(static_cast<size_t>(n_pairs));
  by_sums(ws, n_pairs, p + 4, [&](PairRange pr) {
    const int k = pr.end - pr.first;
    ctx->launches += 2;
    with_p(p, [&](auto pm) {
      glm_pair_sums_kernel<decltype(pm)::value><<<static_cast<unsigned>((k + 7) / 8), 256, 0, ctx->stream>>>(
          g.rows(), g.col.p, g.n, g.kept.p, g.mu.p, ws.glm_w.p, ws.glm_r.p, ctx->pheno.X.p, p, ws.ref_pairs.p, pr,
          ws.ref_sums.p);
    });
    glm_pair_stats_kernel<<<static_cast<unsigned>((k + 63) / 64), 64, 0, ctx->stream>>>(
        ws.ref_sums.p, g.n, p, ws.ainv.p, ws.glm_ok.p, ws.ref_pairs.p, pr, ws.refined.p);
    EQTL_CUDA(cudaGetLastError());
  });
}

void scan_glm(eqtl_ctx* ctx, const eqtl_scan_params* prm, const double* Y, const double* X, double* phi_out,
              uint8_t* converged_out, eqtl_gene_result* genes, PairList& pairs, PairList& cands) {
  Geno& g = ctx->geno;
  Workspace& ws = ctx->ws;
  const int n = prm->n, G = prm->n_genes, p = prm->p;
  EQTL_CHECK(g.m_all > 0, EQTL_E_STATE, "scan_glm: no genotypes loaded");
  EQTL_CHECK(!g.subset, EQTL_E_UNSUPPORTED, "scan_glm: the NB-GLM scan takes every analysis sample");
  EQTL_CHECK(n == g.n, EQTL_E_ARG, "scan_glm: n differs from the loaded genotypes");
  EQTL_CHECK(G > 0, EQTL_E_ARG, "scan_glm: no genes");
  EQTL_CHECK(g.m < (int64_t(1) << 30), EQTL_E_UNSUPPORTED, "scan_glm: more than 2^30 kept SNPs");
  EQTL_CHECK(p >= 1 && p <= kMaxPLmm, EQTL_E_UNSUPPORTED,
             "the GLM scan handles 1 to 32 covariate columns (intercept included)");
  EQTL_CHECK(ctx->precision == EQTL_PREC_SPLIT_F16, EQTL_E_UNSUPPORTED, "the GLM scan runs split-FP16");
  const bool grouped = p > 2;
  cudaStream_t st = ctx->stream;
  const PhenoDev& ph = resolve_pheno(ctx, prm, Y, X);
  std::unique_ptr<StageScope> prep_timer(new StageScope(ctx, EQTL_STAGE_PREP));
  // ---- null fits
  const size_t gn = static_cast<size_t>(G) * n;
  ws.glm_mu.alloc(gn);
  ws.glm_w.alloc(gn);
  ws.glm_r.alloc(gn);
  ws.glm_phi.alloc(G);
  ws.glm_rsum.alloc(G);
  ws.glm_ok.alloc(G);
  ws.glm_counts.alloc(G);
  ws.ainv.alloc(static_cast<size_t>(G) * p * p);
  ++ctx->launches;
  glm_null_kernel<<<G, kGlmThreads, 0, st>>>(ph.Y.p, ph.X.p, n, p, G, ws.glm_mu.p, ws.glm_w.p, ws.glm_r.p,
                                             ws.glm_phi.p, ws.ainv.p, ws.glm_rsum.p, ws.glm_ok.p, ws.glm_counts.p);
  EQTL_CUDA(cudaGetLastError());
  {
    std::vector<uint8_t> counts(G), ok(G);
    ws.glm_counts.download(counts.data(), G, st);
    ws.glm_ok.download(ok.data(), G, st);
    if (phi_out) ws.glm_phi.download(phi_out, G, st);
    EQTL_CUDA(cudaStreamSynchronize(st));
    for (int j = 0; j < G; ++j)
      EQTL_CHECK(counts[j], EQTL_E_ARG, "glm (NB) requires non-negative integer counts (column " + std::to_string(j) + ")");
    if (converged_out) std::copy(ok.begin(), ok.end(), converged_out);
  }
  // ---- SNP-side operands (unrotated), means and gene-side operands
  Rotated& S = ctx->glm_ops;
  const int k_pad = g.k_pad;
  const int64_t m = g.m;
  float s1, s2;
  output_scales(n, s1, s2);
  if (!(S.m == m && S.k_pad == k_pad && S.gt_hi.p)) {
    const size_t elems = static_cast<size_t>(m) * k_pad;
    S.gt_hi.alloc(elems);
    S.gt_lo.alloc(elems);
    S.gt2_hi.alloc(elems);
    S.gt2_lo.alloc(elems);
    if (elems) {
      ++ctx->launches;
      glm_snp_ops_kernel<<<static_cast<unsigned>(std::min<int64_t>((elems + 255) / 256, 148 * 64)), 256, 0, st>>>(
          g.gc_hi.p, g.gc_lo.p, static_cast<int64_t>(elems), 1.0 / kGcScale, s1, s2, S.gt_hi.p, S.gt_lo.p,
          S.gt2_hi.p, S.gt2_lo.p);
      EQTL_CUDA(cudaGetLastError());
    }
    S.m = m;
    S.k_pad = k_pad;
  }
  const int64_t padded = ((m + 255) / 256 + 1) * 256;
  ws.snp_mean.alloc(static_cast<size_t>(std::max<int64_t>(padded, G)));
  ws.glm_rsum_f.alloc(G);
  ++ctx->launches;
  glm_means_kernel<<<static_cast<unsigned>(std::min<int64_t>((std::max<int64_t>(padded, G) + 255) / 256, 4096)), 256,
                     0, st>>>(g.kept.p, m, g.mu.p, std::max<int64_t>(padded, G), ws.snp_mean.p, ws.glm_rsum.p, G,
                              ws.glm_rsum_f.p);
  EQTL_CUDA(cudaGetLastError());
  const int nops = p + 2;
  std::vector<__half*> oph(2 * nops);
  for (int k = 0; k < nops; ++k) {
    ws.ops_hi[k].alloc(static_cast<size_t>(G) * k_pad);
    ws.ops_lo[k].alloc(static_cast<size_t>(G) * k_pad);
    oph[k] = ws.ops_hi[k].p;
    oph[nops + k] = ws.ops_lo[k].p;
  }
  ws.ops_ptr.upload(oph.data(), oph.size(), st);
  ws.unscale.alloc(static_cast<size_t>(G) * nops);
  const GeneOrder go = gene_order(ctx, prm);
  ++ctx->launches;
  glm_gene_ops_kernel<<<G, 256, 0, st>>>(ws.glm_w.p, ws.glm_r.p, ph.X.p, ws.ainv.p, n, p, G, go.row, k_pad, s1, s2,
                                         grouped ? 1 : 0, ws.ops_ptr.p, ws.ops_ptr.p + nops, ws.unscale.p);
  EQTL_CUDA(cudaGetLastError());
  lmm_gate(ctx);
  const Windows win =
      upload_windows(ctx, prm, m, prm->exclude_cis == 2 ? kWinInclude : prm->exclude_cis ? kWinExclude : kWinNone);
  double z_cand = z_critical(prm->pthr);
  if (prm->perm_thr > 0) z_cand = std::min(z_cand, z_critical(prm->perm_thr));
  const TTable tt = device_ttable(ctx, 0.0, true);
  prep_timer.reset();
  // ---- scan
  ScanOutputs so(ctx, G, m, expected_candidates(prm, m));
  const int2* tiles = nullptr;
  int n_tiles = 0;
  cis_tile_list(ctx, win, G, go, m, grouped ? GlmGroupEpi::kTileN : 128, tiles, n_tiles);
  std::unique_ptr<StageScope> scan_timer(new StageScope(ctx, EQTL_STAGE_SCAN));
  if (m > 0 && grouped) {
    GlmGroupEpiParams ep{};
    ep.G = G;
    ep.order = go.gene;
    ep.m = m;
    ep.n_acc = nops;
    ep.unscale = ws.unscale.p;
    ep.snp_ok = ws.ok.p;
    ep.win = win;
    ep.t_cand = static_cast<float>(z_cand * (1.0 - 1e-3));
    ep.tt = tt;
    ep.snp_mean = ws.snp_mean.p;
    ep.rsum = ws.glm_rsum_f.p;
    ep.gene_ok = ws.glm_ok.p;
    const __half* bh[2] = {S.gt_hi.p, S.gt2_hi.p};
    const __half* bl[2] = {S.gt_lo.p, S.gt2_lo.p};
    so.run([&](GeneOut out) {
      ep.out = out;
      launch_grouped(ctx, false, ep, oph.data(), nops, G, bh, bl, S.m, S.k_pad, tiles, n_tiles);
    });
  } else if (m > 0) {
    const __half* ah[4] = {oph[0], oph[1], oph[2], nops > 3 ? oph[3] : oph[2]};
    const __half* al[4] = {oph[nops + 0], oph[nops + 1], oph[nops + 2], nops > 3 ? oph[nops + 3] : oph[nops + 2]};
    auto fill = [&](auto& ep) {
      ep.G = G;
      ep.order = go.gene;
      ep.m = m;
      ep.unscale = ws.unscale.p;
      ep.ainv = ws.ainv.p;
      ep.snp_ok = ws.ok.p;
      ep.win = win;
      ep.t_cand = static_cast<float>(z_cand * (1.0 - 1e-3));
      ep.tt = tt;
      ep.snp_mean = ws.snp_mean.p;
      ep.rsum = ws.glm_rsum_f.p;
      ep.gene_ok = ws.glm_ok.p;
    };
    if (p == 1) {
      GlmEpiParams<1> ep{};
      fill(ep);
      so.run([&](GeneOut out) {
        ep.out = out;
        lmm_launch<1>(ctx, ep, ah, al, G, false, tiles, n_tiles, S);
      });
    } else {
      GlmEpiParams<2> ep{};
      fill(ep);
      so.run([&](GeneOut out) {
        ep.out = out;
        lmm_launch<2>(ctx, ep, ah, al, G, false, tiles, n_tiles, S);
      });
    }
  }
  scan_timer.reset();
  so.collect();
  // ---- FP64 refinement of the candidates, deferred and tiny-|z| pairs
  StageScope refine_timer(ctx, EQTL_STAGE_REFINE);
  glm_refine_pairs(ctx, p, so.n_todo);
  so.finish(prm, genes, pairs, cands);
}

}  // namespace eqtl
