// Device bodies of the panel, solve and reduction kernels, shared by the
// single-problem kernels (potrf.cu) and the batched kernels (batch.cu).  Each
// body works on one tile (or one 64x64 block) given by pointers, so a kernel
// only has to locate its tile.
#pragma once
#include "common.cuh"

namespace egs {

constexpr int kNB = 64;  // inner block width of the panel factorisation

__device__ __forceinline__ double block_sum_256(double v, double* red) {
  red[threadIdx.x] = v;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  const double out = red[0];
  __syncthreads();
  return out;
}

// zi -= T zk for the 64 rows of block rblk of tile T (256 threads = 64 rows x
// 4 column groups, fixed reduction order, FP64 arithmetic whatever the tile's
// storage type).  Dynamic shared memory: ts doubles.
template <typename Tile>
__device__ __forceinline__ void gemv_panel_body(const Tile* __restrict__ T, int ts, const double* __restrict__ zk,
                                                double* __restrict__ zi, int rblk) {
  extern __shared__ double zks[];  // ts
  __shared__ double red[4][kNB];
  for (int c = threadIdx.x; c < ts; c += blockDim.x) zks[c] = zk[c];
  __syncthreads();
  const int rl = threadIdx.x % kNB, g = threadIdx.x / kNB;
  const int r = rblk * kNB + rl;
  double acc = 0.0;
  if (r < ts) {
    for (int c = g; c < ts; c += 4) acc = fma((double)T[(long long)c * ts + r], zks[c], acc);
  }
  red[g][rl] = acc;
  __syncthreads();
  if (g == 0 && r < ts) zi[r] -= ((red[0][rl] + red[1][rl]) + red[2][rl]) + red[3][rl];
}

// Sum over the first `rows` diagonal entries of tile T of log L_rr (L_rr > 0
// only, dmdet-codelet.cpp:76-77); 256 threads.
__device__ __forceinline__ double logdet_tile_body(const double* __restrict__ T, int ts, int rows) {
  __shared__ double red[256];
  double acc = 0.0;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    const double d = T[(long long)r * ts + r];
    if (d > 0.0) acc += log(d);
  }
  return block_sum_256(acc, red);
}

// result[0..3] = (log-likelihood, log|C|, Z^T C^-1 Z, info) of one problem
// (ChameleonImplementation.cpp:188-192, :257-265); 256 threads, fixed order.
__device__ __forceinline__ void finalize_body(const double* __restrict__ partial, int nt, const double* __restrict__ z,
                                              int n, double* __restrict__ result, const int* __restrict__ info) {
  __shared__ double red[256];
  double acc = 0.0;
  for (int r = threadIdx.x; r < n; r += blockDim.x) acc = fma(z[r], z[r], acc);
  const double dot = block_sum_256(acc, red);
  if (threadIdx.x == 0) {
    double det = 0.0;
    for (int k = 0; k < nt; ++k) det += partial[k];
    const double logdet = 2.0 * det;
    const double pi = 3.141592653589793;
    const double nn = (double)n;
    result[0] = -0.5 * dot - 0.5 * logdet - (double)(nn / 2.0) * log(2.0 * pi);
    result[1] = logdet;
    result[2] = dot;
    result[3] = (double)(info ? *info : 0);
  }
}

}  // namespace egs
