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

// VEC consecutive elements of a column as doubles (one 16-byte load).
__device__ __forceinline__ void load_vec(const double* p, double (&v)[2]) {
  const double2 t = *reinterpret_cast<const double2*>(p);
  v[0] = t.x;
  v[1] = t.y;
}
__device__ __forceinline__ void load_vec(const float* p, double (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x;
  v[1] = t.y;
  v[2] = t.z;
  v[3] = t.w;
}

// zi -= T zk for the 64 rows of block rblk of tile T (ld ts, a multiple of 64), FP64
// arithmetic whatever the tile's storage type: 256 threads, each VEC = 16 bytes of
// rows and every (256 VEC / 64)-th column, eight loads in flight, fixed reduction order.
// Memory-bound; 16-byte loads keep four times the bytes in flight of one element
// per load (mixed solves, N = 20,011: 50 -> 30 us per launch).  Dynamic shared
// memory: ts doubles.
template <typename Tile>
__device__ __forceinline__ void gemv_panel_body(const Tile* __restrict__ T, int ts, const double* __restrict__ zk,
                                                double* __restrict__ zi, int rblk) {
  constexpr int VEC = 16 / (int)sizeof(Tile), GROUPS = 256 * VEC / kNB;
  extern __shared__ double zks[];  // ts
  __shared__ double red[GROUPS][kNB + 2];
  for (int c = threadIdx.x; c < ts; c += blockDim.x) zks[c] = zk[c];
  __syncthreads();
  const int rl = (threadIdx.x % (kNB / VEC)) * VEC, g = threadIdx.x / (kNB / VEC);
  const Tile* col = T + rblk * kNB + rl;
  double acc[VEC] = {};
#pragma unroll 8
  for (int c = g; c < ts; c += GROUPS) {
    double v[VEC];
    load_vec(col + (long long)c * ts, v);
#pragma unroll
    for (int i = 0; i < VEC; ++i) acc[i] = fma(v[i], zks[c], acc[i]);
  }
#pragma unroll
  for (int i = 0; i < VEC; ++i) red[g][rl + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < kNB) {
    double s = red[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < GROUPS; ++q) s += red[q][threadIdx.x];
    zi[rblk * kNB + threadIdx.x] -= s;
  }
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
