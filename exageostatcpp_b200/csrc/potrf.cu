// Panel-level building blocks of the tiled Cholesky path on sm_100a: the 64-column
// panel step (diagonal block, row solve and update in one launch) and the
// deterministic reductions that turn the factor into the log-likelihood.
//
// Reference counterparts:
//   CHAMELEON_dpotrf_Tile            ChameleonDense.cpp:25-37   (panel part; the trailing
//                                                                update is dgemm_tma.cu)
//   CHAMELEON_dtrsm_Tile (Z := L^-1 Z) ChameleonImplementation.cpp:337-347
//   DMDETCodelet::core_dmdet          dmdet-codelet.cpp:73-80   (sum of log L_kk, L_kk > 0)
//   DDOTPCodelet::cl_ddotp_function   ddotp-codelet.cpp:63-72   (Z^T Z)
//   log-likelihood assembly           ChameleonImplementation.cpp:257-265
//   DMSECodelet                       dmse-codelet.cpp:60-73    (sum (zhat - z)^2)
// Every reduction uses a fixed summation order, so a result does not depend on
// what else runs on the GPU.
#include <cmath>
#include "common.cuh"
#include "kernels.cuh"
#include "panel_bodies.cuh"
#include "panel_step.cuh"

namespace egs {

// One 64-column step of a panel (panel_step_body), and the flush of the step
// before it: blocks [0, steps) are the step's row chunks, the others copy the
// scratch slot of the previous step to its place.  CTAS per SM: one leaves the
// pivot warp enough registers (two cap them at 128 and spill), two take up to 296
// chunks in one wave.  The line is where one CTA per SM needs a second wave, more
// chunks than SMs: first and second step of an outer block at 140 to 148 chunks, 17.3
// and 13.3 us with one per SM, 19.2 and 13.8 with two; at 150 to 174, 30.3 and 21.8
// against 29.6 and 17.0 (launch times; panels of N = 16,000, tile 320, up to 246
// chunks: 6.52 -> 6.19 ms, of N = 40,000, up to 624: 47.0 -> 44.3 ms).
template <int CTAS>
__global__ void __launch_bounds__(kStepThreads, CTAS)
panel_step_kernel(double* col, int ts, int nchunk, int kb, int nb, int gcol, int* info, double* z,
                  double* __restrict__ out, const double* __restrict__ pslot, double* pcol, int pkb, double* pz) {
  extern __shared__ __align__(16) double step_smem[];
  const int steps = nchunk > 0 ? nchunk : 1;
  const int b = blockIdx.x;
  if (b < steps) {
    panel_step_body(step_smem, col, ts, nchunk > 0 ? b : -1, kb, nb, gcol, b == 0 ? info : nullptr, z, out);
  } else {
    panel_flush_body(pslot, pcol, ts, pkb, b - steps, pz);
  }
}

__global__ void __launch_bounds__(kStepThreads)
panel_flush_kernel(const double* __restrict__ slot, double* __restrict__ col, int ts, int kb, double* __restrict__ z) {
  grid_dependents_launch();
  grid_dependency_wait();
  panel_flush_body(slot, col, ts, kb, blockIdx.x, z);
}

long long panel_scratch_doubles() { return kScratchDoubles; }

int launch_panel_step(double* col, int ts, int rows_below, int kb, int nb, int gcol, int* info, double* z,
                      PanelChain& ch, cudaStream_t st) {
  static std::once_flag done[64];
  once_per_device(done, []() {
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(panel_step_kernel<1>, attr, panel_step_smem(kStepMaxBlocks - 1));
    cudaFuncSetAttribute(panel_step_kernel<2>, attr, panel_step_smem(kStepMaxBlocks - 1));
  });
  const int nchunk = rows_below / kStep;
  double* out = ch.scratch + (long long)ch.parity * kScratchSlot;
  const double* pslot = ch.scratch + (long long)(ch.parity ^ 1) * kScratchSlot;
  const int grid = (nchunk > 0 ? nchunk : 1) + ch.chunks;
  auto kern = nchunk > gemm_num_sms() ? panel_step_kernel<2> : panel_step_kernel<1>;
  kern<<<grid, kStepThreads, panel_step_smem(nb), st>>>(col, ts, nchunk, kb, nb, gcol, info, z, out, pslot, ch.col,
                                                        ch.kb, ch.z);
  ch.col = col;
  ch.kb = kb;
  ch.chunks = 1 + (nb < nchunk ? nb : nchunk);
  ch.z = z;
  ch.ts = ts;
  ch.parity ^= 1;
  return launch_status("panel_step_kernel");
}

int launch_panel_flush(PanelChain& ch, cudaStream_t st) {
  if (ch.chunks == 0) return EGS_OK;
  const double* slot = ch.scratch + (long long)(ch.parity ^ 1) * kScratchSlot;
  const int chunks = ch.chunks;
  ch.chunks = 0;
  return launch_overlapped("panel_flush_kernel", panel_flush_kernel, dim3(chunks), dim3(kStepThreads), 0, st, slot,
                           ch.col, ch.ts, ch.kb, ch.z);
}

// ---------------------------------------------------------------------------
// Deterministic reductions.
// ---------------------------------------------------------------------------
// partial[k] = sum over the real rows of diagonal tile k of log L_rr.
__global__ void __launch_bounds__(256)
logdet_partials_kernel(const double* __restrict__ tiles, int ts, int nt, int n, double* __restrict__ partial) {
  const int k = blockIdx.x;
  const int rows = min(ts, n - k * ts);
  grid_dependents_launch();
  grid_dependency_wait();
  const double s = logdet_tile_body(tiles + tile_slot(k, k, nt) * (long long)ts * ts, ts, rows);
  if (threadIdx.x == 0) partial[k] = s;
}

int launch_logdet_partials(const double* tiles, int ts, int nt, int n, double* partial, cudaStream_t st) {
  return launch_overlapped("logdet_partials_kernel", logdet_partials_kernel, dim3(nt), dim3(256), 0, st,
                           tiles, ts, nt, n, partial);
}

// result = (log-likelihood, log|C|, Z^T C^-1 Z after the solve, info) (finalize_body).
__global__ void __launch_bounds__(256)
finalize_kernel(const double* __restrict__ partial, int nt, const double* __restrict__ z, int n,
                double* __restrict__ result, const int* __restrict__ info) {
  grid_dependency_wait();
  finalize_body(partial, nt, z, n, result, info);
}

int launch_finalize(const double* partial, int nt, const double* z, int n, double* result, const int* info,
                    cudaStream_t st) {
  return launch_overlapped("finalize_kernel", finalize_kernel, dim3(1), dim3(256), 0, st, partial, nt, z, n, result,
                           info);
}

// out[0] = sum (a - b)^2 (DMSECodelet, dmse-codelet.cpp:60-73), fixed order.
__global__ void __launch_bounds__(256)
sumsq_diff_kernel(const double* __restrict__ a, const double* __restrict__ b, int n, double* __restrict__ out) {
  __shared__ double red[256];
  double acc = 0.0;
  for (int r = threadIdx.x; r < n; r += blockDim.x) {
    const double d = a[r] - b[r];
    acc = fma(d, d, acc);
  }
  const double s = block_sum_256(acc, red);
  if (threadIdx.x == 0) out[0] = s;
}

void launch_sumsq_diff(const double* a, const double* b, int n, double* out, cudaStream_t st) {
  sumsq_diff_kernel<<<1, 256, 0, st>>>(a, b, n, out);
}

}  // namespace egs

namespace egs {

// out[j] = sum_i A[i + j*lda] * w[i] for j < cols (A is rows x cols column-major):
// the kriging product Zmiss = C12 * Zobs with C12 stored transposed (obs x miss,
// LinearAlgebraMethods.cpp:552).  One warp per output, fixed reduction order.
__global__ void __launch_bounds__(256)
gemv_t_block_kernel(const double* __restrict__ a, long long lda, int rows, int cols, const double* __restrict__ w,
                    double* __restrict__ out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x * 8 + warp;
  if (j >= cols) return;
  const double* col = a + (long long)j * lda;
  double acc = 0.0;
  for (int i = lane; i < rows; i += 32) acc = fma(col[i], w[i], acc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) out[j] = acc;
}

void launch_gemv_t_block(const double* a, long long lda, int rows, int cols, const double* w, double* out,
                         cudaStream_t st) {
  if (cols <= 0) return;
  gemv_t_block_kernel<<<(cols + 7) / 8, 256, 0, st>>>(a, lda, rows, cols, w, out);
}

}  // namespace egs

namespace egs {

// part[slot(i, j)][r] = sum_c L_ij[r][c] e_j[c] over the stored lower tiles (only
// c <= r inside a diagonal tile): the tile products of Z = L e
// (dtrmm in GenerateObservationsVector, LinearAlgebraMethods.cpp:400).
__global__ void __launch_bounds__(256)
trmv_tile_kernel(const double* __restrict__ tiles, int ts, int nt, const double* __restrict__ e,
                 double* __restrict__ part) {
  __shared__ double red[4][kNB];
  const long long slot = blockIdx.y;
  // slot -> (i, j)
  int j = 0;
  while (j < nt - 1 && tile_slot(j + 1, j + 1, nt) <= slot) ++j;
  const int i = j + (int)(slot - tile_slot(j, j, nt));
  const double* T = tiles + slot * (long long)ts * ts;
  const double* ej = e + (long long)j * ts;
  const int rl = threadIdx.x % kNB, g = threadIdx.x / kNB;
  const int r = blockIdx.x * kNB + rl;
  double acc = 0.0;
  if (r < ts) {
    const int cend = (i == j) ? r + 1 : ts;
    for (int c = g; c < cend; c += 4) acc = fma(T[(long long)c * ts + r], ej[c], acc);
  }
  red[g][rl] = acc;
  __syncthreads();
  if (g == 0 && r < ts) part[slot * ts + r] = ((red[0][rl] + red[1][rl]) + red[2][rl]) + red[3][rl];
}

// z[i*ts + r] = sum_{j <= i} part[slot(i, j)][r], j ascending (fixed order).
__global__ void __launch_bounds__(256)
trmv_reduce_kernel(const double* __restrict__ part, int ts, int nt, double* __restrict__ z) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long long)nt * ts) return;
  const int i = (int)(g / ts), r = (int)(g - (long long)i * ts);
  double acc = 0.0;
  for (int j = 0; j <= i; ++j) acc += part[tile_slot(i, j, nt) * ts + r];
  z[g] = acc;
}

void launch_trmv(const double* tiles, int ts, int nt, const double* e, double* part, double* z, cudaStream_t st) {
  const long long nslots = lower_tiles(nt);  // <= 65535 is checked by the caller
  trmv_tile_kernel<<<dim3((ts + kNB - 1) / kNB, (unsigned)nslots), 256, 0, st>>>(tiles, ts, nt, e, part);
  const long long total = (long long)nt * ts;
  trmv_reduce_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(part, ts, nt, z);
}

}  // namespace egs
