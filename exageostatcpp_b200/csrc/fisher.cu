// Fisher information of the Matern parameters on the GPU.
//
// The reference (LinearAlgebraMethods<T>::ExaGeoStatFisherTile,
// src/linear-algebra-solvers/LinearAlgebraMethods.cpp:1133-1306) forms
//     A_jk = 1/2 tr(C^-1 C_j C^-1 C_k),   C_j = dC/dtheta_j,
// with two triangular solves per derivative and one dense product plus a
// trace per pair, and returns A^-1.  Here the same quantity is computed as
//     A_jk = 1/2 sum(M_j o M_k),   M_j = L^-1 C_j L^-T  (symmetric),
// which needs no N^3 product per pair.  C is factored once; the rows of the three
// symmetric C_j, stacked, go through two row solves: X_j = C_j L^-T, then X_j^T L^-T =
// L^-1 C_j L^-T = M_j, of which only the lower half is computed, a third of a full
// solve's work (solve.cu; N = 1,600: second sweep 1.02 -> 0.53 ms, the call 2.96 -> 2.54).
//
// Derivative kernels (src/kernels/concrete/UnivariateMaternDdsigmaSquare.cpp,
// UnivariateMaternDbeta.cpp, UnivariateMaternDnu.cpp): at scaled distance
// x = d / beta > 0, with c = 1 / (2^(nu-1) Gamma(nu)),
//     dC/dsigma2 = c x^nu K_nu(x)                                 (1 at x = 0)
//     dC/dbeta   = sigma2 c [-nu/beta x^nu K_nu - x^nu (nu/x K_nu - K_nu+1) x/beta]
//     dC/dnu     = sigma2 [-2 ln2 2^-nu / Gamma(nu) x^nu K_nu + 2^(1-nu) (-psi(nu)/Gamma(nu) x^nu K_nu
//                          + (x^nu ln x K_nu + x^nu dK_nu/dnu) / Gamma(nu))]  (0 at x = 0).
// The reference differentiates K_nu in nu by a forward difference with step
// 1e-9 (src/helpers/BasselFunction.cpp:23-33); here F_nu(x) = x^nu K_nu(x) itself is
// differentiated: the last two terms are dF/dnu, from the six-point central
// difference with step h = 2e-3 (truncation h^6 / 140 d^7F/dnu^7), and
// dC/dbeta = sigma2 c (F_nu+1 - 2 nu F_nu) / beta.  F comes from the generator's
// tables (e^x F, one per order), where the direct series and continued fraction
// cost thousands of operations for every order (N = 1,600: derivatives 2.7 ms of
// direct evaluations, 0.1 from the tables).
#include <cmath>
#include <memory>
#include <vector>
#include "common.cuh"
#include "kernels.cuh"

namespace egs {

struct FisherParams {
  double sigma2, beta, nu;
  double con;    // 1 / (2^(nu-1) Gamma(nu))
  double psi;    // digamma(nu)
};

// Orders whose F the derivatives need: nu, nu + 1, nu +- h, nu +- 2 h, nu +- 3 h.
constexpr int kFisherOrders = 8;
constexpr double kFisherStep = 2e-3;
constexpr int kFisherTabBytes = kFisherOrders * kKtabShared * (int)sizeof(double);

// F_nu(x) = x^nu K_nu(x) of the order of p (kind 2), from its table where x lies in it.
__device__ __forceinline__ double bessel_f(double x, bool in_table, int idx, double t, double ex,
                                           const MaternParams& p, const double* __restrict__ tab) {
  if (in_table && p.table) return ktab_sum(tab + idx * kKtabRow, t) * ex;
  bool scaled;
  const double k = bessel_k_general(x, p, scaled);
  return pow(x, p.nu) * (scaled ? k * ex : k);
}

// The three derivative matrices stacked as rows, column-major with column stride
// 3 np (rows / columns past n are zero): d[c * 3 np + j * np + r].
__global__ void __launch_bounds__(256)
matern_derivatives_kernel(const double* __restrict__ x, const double* __restrict__ y, int n, int np,
                          FisherParams q, const MaternParams* __restrict__ orders, const double* __restrict__ tabs,
                          double* __restrict__ d) {
  extern __shared__ __align__(16) double stab[];  // kFisherTabBytes
  for (int i = threadIdx.x; i < kFisherOrders * kKtabDoubles; i += 256)
    stab[(i / kKtabStride) * kKtabRow + i % kKtabStride] = tabs[i];
  __syncthreads();
  const long long nn = (long long)np * np;
  for (long long idx = (long long)blockIdx.x * 256 + threadIdx.x; idx < nn; idx += (long long)gridDim.x * 256) {
    const int c = (int)(idx / np), r = (int)(idx - (long long)c * np);
    double ds = 0.0, db = 0.0, dn = 0.0;
    if (r < n && c < n) {
      const double e = euclid_dist(x[r], y[r], x[c], y[c]) / q.beta;
      if (e == 0.0) {
        ds = 1.0;
      } else {
        int at = 0;
        double t = 0.0;
        const bool in_table = ktab_locate(e, at, t);
        const double ex = exp(-e);
        double f[kFisherOrders];
#pragma unroll
        for (int o = 0; o < kFisherOrders; ++o)
          f[o] = bessel_f(e, in_table, at, t, ex, orders[o], stab + o * kKtabShared);
        const double df = (45.0 * (f[2] - f[3]) - 9.0 * (f[4] - f[5]) + (f[6] - f[7])) / (60.0 * kFisherStep);
        ds = q.con * f[0];
        db = q.sigma2 * q.con / q.beta * (f[1] - 2.0 * q.nu * f[0]);
        dn = q.sigma2 * q.con * (df - (log(2.0) + q.psi) * f[0]);
      }
    }
    double* out = d + (long long)c * 3 * np + r;
    out[0] = ds;
    out[np] = db;
    out[2 * (long long)np] = dn;
  }
}

// Y_j := X_j^T for the three stacked np x np matrices (64 x 64 blocks through
// shared memory).
__global__ void __launch_bounds__(256)
transpose_stacked_kernel(const double* __restrict__ X, int np, double* __restrict__ Y) {
  __shared__ double t[64][65];
  const long long ld = 3LL * np;
  const double* src = X + (long long)blockIdx.z * np;
  double* dst = Y + (long long)blockIdx.z * np;
  const int r0 = 64 * blockIdx.x, c0 = 64 * blockIdx.y, r = threadIdx.x & 63;
  for (int c = threadIdx.x >> 6; c < 64; c += 4) t[c][r] = src[(c0 + c) * ld + r0 + r];
  __syncthreads();
  for (int c = threadIdx.x >> 6; c < 64; c += 4) dst[(r0 + c) * ld + c0 + r] = t[r][c];
}

// The six sums of M_j o M_k (j <= k) over the lower halves of the stacked symmetric
// matrices: per-block partial sums in a fixed order, then one warp per pair adds the
// partials in a fixed order.
constexpr int kPairs = 6;
__global__ void __launch_bounds__(256)
pair_dots_kernel(const double* __restrict__ M, int np, double* __restrict__ partial) {
  __shared__ double red[256];
  double acc[kPairs] = {};
  const long long nn = (long long)np * np;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < nn; i += (long long)gridDim.x * 256) {
    const long long c = i / np, r = i - c * np;
    if (r < c) continue;
    const double w = (r == c) ? 1.0 : 2.0;
    const double* m = M + c * 3 * np + r;
    const double a = m[0], b = m[np], d = m[2 * (long long)np];
    const double wa = w * a, wb = w * b;
    acc[0] = fma(wa, a, acc[0]);
    acc[1] = fma(wa, b, acc[1]);
    acc[2] = fma(wa, d, acc[2]);
    acc[3] = fma(wb, b, acc[3]);
    acc[4] = fma(wb, d, acc[4]);
    acc[5] = fma(w * d, d, acc[5]);
  }
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    red[threadIdx.x] = acc[q];
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
      if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x * kPairs + q] = red[0];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(32 * kPairs)
pair_sums_kernel(const double* __restrict__ partial, int m, double* __restrict__ out) {
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0;
  for (int i = lane; i < m; i += 32) s += partial[i * kPairs + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[q] = s;
}

}  // namespace egs

using namespace egs;

namespace {

// digamma(x), x > 0: recurrence psi(x) = psi(x+1) - 1/x up to x >= 16, then the
// asymptotic series ln x - 1/(2x) - sum B_2k / (2k x^2k) (Abramowitz & Stegun
// 6.3.18), whose first omitted term is 0.021 / x^12 < 1e-16.
double digamma(double x) {
  double r = 0.0;
  while (x < 16.0) {
    r -= 1.0 / x;
    x += 1.0;
  }
  const double f = 1.0 / (x * x);
  const double series = f * (1.0 / 12 - f * (1.0 / 120 - f * (1.0 / 252 - f * (1.0 / 240 - f * (1.0 / 132)))));
  return r + std::log(x) - 0.5 / x - series;
}

}  // namespace

namespace egs {
int factor_resident(egs_problem* p, const double* theta);
int problem_tiles(egs_problem* p, double** tiles, double** x, double** y, int* ts, int* nt, cudaStream_t* st);
}  // namespace egs

extern "C" int egs_fisher_host(int n, int dts, const double* x, const double* y, const double* theta,
                               double* fisher_inverse) {
  if (n <= 0 || dts <= 0 || !x || !y || !theta || !fisher_inverse) return EGS_ERR_INVALID;
  MaternParams mp;
  if (make_matern_params(theta, &mp) != EGS_OK) {
    set_last_error("theta outside the Matern domain (sigma2 > 0, beta > 0, nu > 0)", "egs_fisher_host");
    return EGS_ERR_INVALID;
  }
  egs_problem* p = nullptr;
  int rc = egs_problem_create(&p, n, dts);
  if (rc != EGS_OK) return rc;
  std::unique_ptr<egs_problem, int (*)(egs_problem*)> guard(p, egs_problem_destroy);
  double *tiles = nullptr, *dx = nullptr, *dy = nullptr;
  int ts = 0, nt = 0;
  cudaStream_t st = nullptr;
  problem_tiles(p, &tiles, &dx, &dy, &ts, &nt, &st);
  // The sweeps below have no such limit: it is the entry's, kept from the form that
  // factored a matrix of 2 nt tile rows, so that what it refuses does not change.
  if (lower_tiles(2 * nt) > 65535) {
    set_last_error("more than 180 tile rows; use a larger dts", "egs_fisher_host");
    return EGS_ERR_INVALID;
  }
  if ((rc = egs_problem_set_locations(p, x, y)) != EGS_OK || (rc = factor_resident(p, theta)) != EGS_OK) return rc;
  const int np = factor_rows(n);
  const size_t nn3 = 3 * (size_t)np * np;
  double *Y = nullptr, *X = nullptr, *tabs = nullptr, *part = nullptr, *dots = nullptr;
  MaternParams* orders = nullptr;
  const int nblk = 296;
  auto cleanup = [&]() {
    cudaStreamSynchronize(st);
    for (void* b : {(void*)Y, (void*)X, (void*)tabs, (void*)orders, (void*)part, (void*)dots})
      if (b) cudaFreeAsync(b, st);
    cudaStreamSynchronize(st);
  };
  static std::once_flag tab_attr[64];
  once_per_device(tab_attr, []() {
    cudaFuncSetAttribute(matern_derivatives_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFisherTabBytes);
  });
  const struct {
    void** p;
    size_t bytes;
  } bufs[] = {{(void**)&Y, nn3 * sizeof(double)},      {(void**)&X, nn3 * sizeof(double)},
              {(void**)&tabs, (size_t)kFisherTabBytes}, {(void**)&orders, kFisherOrders * sizeof(MaternParams)},
              {(void**)&part, kPairs * nblk * sizeof(double)}, {(void**)&dots, kPairs * sizeof(double)}};
  for (const auto& b : bufs)
    if (alloc_from_pool(b.p, b.bytes, st) != EGS_OK) {
      cleanup();
      set_last_error("device allocation failed", "egs_fisher_host");
      return EGS_ERR_OOM;
    }
  FisherParams q;
  q.sigma2 = theta[0];
  q.beta = theta[1];
  q.nu = theta[2];
  q.con = 1.0 / (std::pow(2.0, q.nu - 1.0) * std::tgamma(q.nu));
  q.psi = digamma(q.nu);
  // every order as a general one (half-integers included: mu = -1/2); orders
  // below 0 (nu < 6e-3) mean K_{-nu} = K_nu
  const double h = kFisherStep;
  const double order[kFisherOrders] = {q.nu,           q.nu + 1.0,     q.nu + h,       q.nu - h,
                                       q.nu + 2.0 * h, q.nu - 2.0 * h, q.nu + 3.0 * h, q.nu - 3.0 * h};
  MaternParams hp[kFisherOrders];
  for (int o = 0; o < kFisherOrders; ++o) {
    hp[o] = mp;
    hp[o].nu = order[o];
    hp[o].n = (int)std::floor(order[o] + 0.5);
    hp[o].mu = order[o] - hp[o].n;
    hp[o].kind = 2;
    hp[o].table = q.nu + 1.0 <= kKtabMaxNu ? 1 : 0;
  }
  cudaMemcpyAsync(orders, hp, sizeof(hp), cudaMemcpyHostToDevice, st);
  launch_matern_ktab(orders, tabs, kFisherOrders, st);
  matern_derivatives_kernel<<<3 * gemm_num_sms(), 256, kFisherTabBytes, st>>>(dx, dy, n, np, q, orders, tabs, Y);
  // Y = C_j -> X = C_j L^-T; Y = X^T = L^-1 C_j -> X = L^-1 C_j L^-T = M_j, its lower half
  if ((rc = launch_rows_forward(tiles, ts, nt, np / 64, Y, X, 3LL * np, 3 * np, st)) != EGS_OK) {
    cleanup();
    return rc;
  }
  transpose_stacked_kernel<<<dim3(np / 64, np / 64, 3), 256, 0, st>>>(X, np, Y);
  if ((rc = launch_rows_forward_symmetric(tiles, ts, nt, np / 64, Y, X, 3, st)) != EGS_OK) {
    cleanup();
    return rc;
  }
  pair_dots_kernel<<<nblk, 256, 0, st>>>(X, np, part);
  pair_sums_kernel<<<1, 32 * kPairs, 0, st>>>(part, nblk, dots);
  double h6[kPairs] = {};
  cudaMemcpyAsync(h6, dots, sizeof(h6), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    set_last_error("a CUDA call failed", "egs_fisher_host");
    cleanup();
    return EGS_ERR_CUDA;
  }
  cleanup();
  // A (3 x 3, symmetric) and its inverse through a Cholesky factorisation
  double A[3][3];
  for (int j = 0, i = 0; j < 3; ++j)
    for (int k = j; k < 3; ++k) A[j][k] = A[k][j] = 0.5 * h6[i++];
  double L[3][3] = {};
  for (int j = 0; j < 3; ++j) {
    double s = A[j][j];
    for (int k = 0; k < j; ++k) s -= L[j][k] * L[j][k];
    if (!(s > 0.0)) {
      set_last_error("Fisher information not positive definite", "egs_fisher_host");
      return j + 1;
    }
    L[j][j] = std::sqrt(s);
    for (int i = j + 1; i < 3; ++i) {
      double t = A[i][j];
      for (int k = 0; k < j; ++k) t -= L[i][k] * L[j][k];
      L[i][j] = t / L[j][j];
    }
  }
  for (int c = 0; c < 3; ++c) {  // column c of A^-1: L L^T v = e_c
    double v[3] = {0, 0, 0};
    v[c] = 1.0;
    for (int i = 0; i < 3; ++i) {
      for (int k = 0; k < i; ++k) v[i] -= L[i][k] * v[k];
      v[i] /= L[i][i];
    }
    for (int i = 2; i >= 0; --i) {
      for (int k = i + 1; k < 3; ++k) v[i] -= L[k][i] * v[k];
      v[i] /= L[i][i];
    }
    for (int i = 0; i < 3; ++i) fisher_inverse[c * 3 + i] = v[i];
  }
  return EGS_OK;
}
