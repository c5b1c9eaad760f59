// Triangular solves against a finished lower tiled factor, sm_100a.
//
// One right-hand side (vec_*): one launch per 64 columns.  Every CTA owns 64 rows
// (forward) or 64 columns (backward) of the remaining vector, solves the 64 x 64 diagonal
// block itself and applies its own 64 x 64 block of L.  The factor does not
// depend on the vector, so a CTA fetches both blocks before it waits for the
// previous step (programmatic dependent launch): only the vector's chain of 64
// unknowns per step is serial.  Bound by that chain, about 4 us per step; one
// 1,024-thread CTA per tile with the blocks fetched in the chain, and a launch for the
// rest of the tile row, took 35 to 45 us per 64 unknowns.
//
// Many right-hand sides (rows_*): the vectors are the rows of a matrix Y (row q
// at Y[c * ldy + q]), so that forward is Y L^-T and backward Y L^-1, a row solve per
// 64 x 64 block and DMMA updates as in the panel step.  Solved columns go to a
// second matrix: every CTA of a step reads the unsolved ones.
//
// Reference counterparts: CHAMELEON_dtrsm_Tile / dposv on one vector
// (ChameleonImplementation.cpp:337-347, LinearAlgebraMethods.cpp:544) and the
// per-target solves of the MLOE / MMOM loop (LinearAlgebraMethods.cpp:802-1131).
#include <algorithm>
#include "common.cuh"
#include "kernels.cuh"
#include "panel_step.cuh"

namespace egs {

namespace {

constexpr int kVecThreads = 256;

// The 64 x 64 block at `src` (column stride ts) into shared memory.
__device__ __forceinline__ void load_block(double* dst, const double* src, long long ld, int threads) {
  for (int e = threadIdx.x; e < kStep * kStep / 2; e += threads) {
    const int c = e >> 5, r = 2 * (e & 31);
    cp_async16(dst + c * kStepLd + r, src + c * ld + r);
  }
}

// One warp: x := L^-1 x (kBack: L^-T x) for 64 unknowns in shared memory, eight
// at a time: every lane solves the 8 x 8 block in registers, then lane r updates
// rows r and r + 32.  pinv holds 1 / L_jj.
template <bool kBack>
__device__ __forceinline__ void vec_solve64(const double* D, const double* pinv, double* x, int lane) {
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    const int b = kBack ? 7 - i : i;
    const double* blk = D + (8 * b) * kStepLd + 8 * b;
    double v[8];
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 p = *reinterpret_cast<const double2*>(x + 8 * b + c);
      v[c] = p.x;
      v[c + 1] = p.y;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = kBack ? 7 - u : u;
      v[j] *= pinv[8 * b + j];
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (kBack ? c < j : c > j) v[c] = fma(-(kBack ? blk[c * kStepLd + j] : blk[j * kStepLd + c]), v[j], v[c]);
    }
    double y0 = x[lane], y1 = x[lane + 32];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int o = kBack ? 8 * b + q : (8 * b + q) * kStepLd;
      y0 = fma(-D[o + (kBack ? lane * kStepLd : lane)], v[q], y0);
      y1 = fma(-D[o + (kBack ? (lane + 32) * kStepLd : lane + 32)], v[q], y1);
    }
    __syncwarp();
    const int own = lane >> 3;  // the block's own rows get the solution, later ones the update
    if (kBack ? own < b : own > b) x[lane] = y0;
    if (kBack ? own + 4 < b : own + 4 > b) x[lane + 32] = y1;
    if (lane < 8) {
      double s = v[0];
#pragma unroll
      for (int c = 1; c < 8; ++c) s = (lane == c) ? v[c] : s;
      x[8 * b + lane] = s;
    }
    __syncwarp();
  }
}

// Step of the 64 unknowns at global row r0 (tile k, local column kb).  Block b:
// forward, rows r0 + 64 (b + 1) ..; backward, columns 64 b .. (rows / columns of
// the vector).  Block 0 also moves the previous step's solution (prev, 64
// values) to pz; this step's goes to out.
template <bool kBack>
__global__ void __launch_bounds__(kVecThreads)
vec_step_kernel(const double* __restrict__ tiles, int ts, int nt, int k, int kb, int nblk, double* z,
                double* __restrict__ out, const double* prev, double* pz) {
  __shared__ __align__(16) double D[kStepBlock];
  __shared__ __align__(16) double x[kStep];
  __shared__ double pinv[kStep];
  __shared__ double red[4][kStep];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long ts2 = (long long)ts * ts;
  const double* diag = tiles + tile_slot(k, k, nt) * ts2 + (long long)kb * ts + kb;
  load_block(D, diag, ts, kVecThreads);
  cp_async_commit();
  // this CTA's block of L: forward row r, columns 16 g .. of the step; backward
  // column r of the block, rows 16 g .. of the step
  const bool have = (int)blockIdx.x < nblk;
  const int r = tid & 63, g = tid >> 6;
  const int at = kBack ? kStep * blockIdx.x : k * ts + kb + kStep * (blockIdx.x + 1);  // first row / column
  double a[16];
  if (have) {
    const int t = at / ts, lo = at - t * ts;
    if (kBack) {
      const double* p = tiles + tile_slot(k, t, nt) * ts2 + (long long)(lo + r) * ts + kb + 16 * g;
#pragma unroll
      for (int i = 0; i < 16; i += 2) ldg_v2f64(p + i, a[i], a[i + 1]);
    } else {
      const double* p = tiles + tile_slot(t, k, nt) * ts2 + (long long)(kb + 16 * g) * ts + lo + r;
#pragma unroll
      for (int i = 0; i < 16; ++i) a[i] = p[(long long)i * ts];
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  if (tid < kStep) pinv[tid] = 1.0 / D[tid * kStepLd + tid];
  grid_dependents_launch();
  grid_dependency_wait();
  if (tid < kStep) x[tid] = z[k * ts + kb + tid];
  const double zi = (have && g == 0) ? z[at + r] : 0.0;
  if (blockIdx.x == 0 && prev && tid >= kVecThreads - kStep) {
    const int i = tid - (kVecThreads - kStep);
    pz[i] = prev[i];
  }
  __syncthreads();
  if (warp == 0) vec_solve64<kBack>(D, pinv, x, lane);
  __syncthreads();
  if (blockIdx.x == 0 && tid < kStep) out[tid] = x[tid];
  if (!have) return;
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    s0 = fma(a[i], x[16 * g + i], s0);
    s1 = fma(a[i + 1], x[16 * g + i + 1], s1);
  }
  red[g][r] = s0 + s1;
  __syncthreads();
  if (g == 0) z[at + r] = zi - (((red[0][r] + red[1][r]) + red[2][r]) + red[3][r]);
}

__global__ void vec_last_kernel(const double* __restrict__ prev, double* __restrict__ pz) {
  grid_dependency_wait();
  pz[threadIdx.x] = prev[threadIdx.x];
}

template <bool kBack>
int vec_solve(const double* tiles, int ts, int nt, int rows, double* z, double* scratch, cudaStream_t st,
              long long* launches) {
  const int per = ts / kStep, steps = rows / kStep;
  const double* prev = nullptr;
  double* pz = nullptr;
  for (int i = 0; i < steps; ++i) {
    const int b = kBack ? steps - 1 - i : i;  // 64-row block of the vector
    const int nblk = kBack ? b : steps - 1 - b;
    double* out = scratch + (i & 1) * kStep;
    // the first step starts after whatever wrote the factor
    int rc = EGS_OK;
    if (i == 0) {
      vec_step_kernel<kBack><<<nblk > 0 ? nblk : 1, kVecThreads, 0, st>>>(tiles, ts, nt, b / per, (b % per) * kStep,
                                                                          nblk, z, out, prev, pz);
      rc = launch_status("vec_step_kernel");
    } else {
      rc = launch_overlapped("vec_step_kernel", vec_step_kernel<kBack>, dim3(nblk > 0 ? nblk : 1), dim3(kVecThreads),
                             0, st, tiles, ts, nt, b / per, (b % per) * kStep, nblk, z, out, prev, pz);
    }
    if (rc != EGS_OK) return rc;
    prev = out;
    pz = z + (long long)b * kStep;
  }
  *launches += steps + 1;
  return launch_overlapped("vec_last_kernel", vec_last_kernel, dim3(1), dim3(kStep), 0, st, prev, pz);
}

// ---------------------------------------------------------------------------
// Many right-hand sides, as rows
// ---------------------------------------------------------------------------
constexpr int kRowsThreads = 128;

// B fragment whose column n is column n0 + n of the column-major block x.
__device__ __forceinline__ void frag_bt(const double* x, int n0, int k0, int lane, double (&b)[4]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) b[i] = x[(n0 + g) * kStepLd + k0 + t + 4 * i];
}

// One warp: rows row0 .. row0+15 of X (the upper lanes repeat the lower ones),
// sub-block q (16 columns) of X := X L^-1: substitution against L_qq from the
// last column down, then the update of the earlier sub-blocks.
__device__ __forceinline__ void rows_back16(double* X, const double* D, const double* pinv, int q, int row0, int lane) {
  double* xr = X + row0 + (lane & 15);
  const double* blk = D + (16 * q) * kStepLd + 16 * q;
  {
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = xr[(16 * q + j) * kStepLd];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int j = 15 - u;
      v[j] *= pinv[16 * q + j];
#pragma unroll
      for (int c = 0; c < 16; ++c)
        if (c < j) v[c] = fma(-v[j], blk[c * kStepLd + j], v[c]);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 16; ++j) xr[(16 * q + j) * kStepLd] = v[j];
  }
  __syncwarp();
  if (q == 0) return;
  double a[8];
  frag_a_neg(X, row0, 16 * q, lane, a);
#pragma unroll 2
  for (int n0 = 0; n0 < 16 * q; n0 += 8) {
    double b[4], c[4];
    frag_bt(D, n0, 16 * q, lane, b);  // rows 16 q .. of columns n0 ..
    frag_c_load(X, row0, n0, lane, c);
    dmma_16816(c, a, b);
    frag_c_store(X, row0, n0, lane, c);
  }
  __syncwarp();
}

// Step of the 64 columns at global column r0 = k ts + kb: X_b := Y_b L_bb^-T (kBack:
// L_bb^-1) for one chunk of 64 rows, and Y_j -= X_b L_jb^T (kBack: X_b L_bj) for the
// remaining column blocks j, share of them per CTA of the row.  Y and X are
// column-major with column stride ldy.  With sym > 0 the rows are stacked symmetric
// results of sym chunks each, of which only the blocks on and below the diagonal are
// wanted: the chunks above block column b are left out, the others stop at theirs.
template <bool kBack>
__global__ void __launch_bounds__(kRowsThreads)
rows_step_kernel(const double* __restrict__ tiles, int ts, int nt, int k, int kb, int nblk, int share, int sym,
                 double* Y, double* __restrict__ X, long long ldy) {
  extern __shared__ __align__(16) double sm[];
  double *D = sm, *A = sm + kStepBlock, *B = sm + 2 * kStepBlock, *pinv = sm + 3 * kStepBlock;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long ts2 = (long long)ts * ts;
  const int r0 = k * ts + kb;
  int chunk = blockIdx.y;
  if (sym > 0) {
    const int left = nblk + 1;  // chunks per matrix from block column b on, the longest first
    chunk = (blockIdx.y / left) * sym + sym - 1 - blockIdx.y % left;
    nblk -= blockIdx.y % left;
  }
  const int step = (nblk + share - 1) / share;  // CTAs with blocks of this row
  if (blockIdx.x > 0 && (int)blockIdx.x >= step) {
    grid_dependency_wait();
    return;
  }
  double* Yc = Y + kStep * chunk;
  auto first_col = [&](int j) { return kBack ? kStep * j : r0 + kStep * (j + 1); };
  auto fetch_b = [&](int j) {
    const int at = first_col(j), t = at / ts, lo = at - t * ts;
    load_block(B, tiles + (kBack ? tile_slot(k, t, nt) * ts2 + (long long)lo * ts + kb
                                 : tile_slot(t, k, nt) * ts2 + (long long)kb * ts + lo),
               ts, kRowsThreads);
  };
  load_block(D, tiles + tile_slot(k, k, nt) * ts2 + (long long)kb * ts + kb, ts, kRowsThreads);
  if ((int)blockIdx.x < nblk) fetch_b(blockIdx.x);
  cp_async_commit();
  // the factor does not change between the steps, so its blocks are under way before
  // the wait for the step that wrote Y (N = 1,600: Fisher 2.53 -> 2.41 ms, MLOE 2.07 -> 2.02)
  grid_dependents_launch();
  grid_dependency_wait();
  load_block(A, Yc + r0 * ldy, ldy, kRowsThreads);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (tid < kStep) pinv[tid] = 1.0 / D[tid * kStepLd + tid];
  __syncthreads();
#pragma unroll 1
  for (int u = 0; u < 4; ++u) {
    if constexpr (kBack) {
      rows_back16(A, D, pinv, 3 - u, 16 * warp, lane);
    } else {
      step_rows<1>(A, D, pinv, u, 16 * warp, lane);
    }
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    double* Xc = X + kStep * chunk;
    for (int e = tid; e < kStep * kStep / 2; e += kRowsThreads) {
      const int c = e >> 5, r = 2 * (e & 31);
      *reinterpret_cast<double2*>(Xc + (r0 + c) * ldy + r) = *reinterpret_cast<const double2*>(A + c * kStepLd + r);
    }
  }
  const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int j = blockIdx.x; j < nblk; j += step) {
    if (j != (int)blockIdx.x) {
      __syncthreads();  // every warp is done with the previous block of L
      fetch_b(j);
      cp_async_commit();
    }
    // this warp's 16 rows of Y_j, under way together with the block of L
    double* p = Yc + (long long)(first_col(j) + 2 * t) * ldy + 16 * warp + 2 * g;
    double c[8][4];
#pragma unroll
    for (int ni = 0; ni < 8; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) ldg_v2f64(p + (8 * ni + h) * ldy, c[ni][h], c[ni][2 + h]);
    if (j != (int)blockIdx.x) {
      cp_async_wait<0>();
      __syncthreads();
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      double a[8];
      frag_a_neg(A, 16 * warp, 16 * kk, lane, a);
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        double b[4];
        if constexpr (kBack) {
          frag_bt(B, 8 * ni, 16 * kk, lane, b);
        } else {
          frag_b(B, 8 * ni, 16 * kk, lane, b);
        }
        dmma_16816(c[ni], a, b);
      }
    }
#pragma unroll
    for (int ni = 0; ni < 8; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) stg_v2f64(p + (8 * ni + h) * ldy, c[ni][h], c[ni][2 + h]);
  }
}

// U(:, j) = -W L(:, j) for the 64-column block j = blockIdx.x and the 64 rows of
// blockIdx.y: sum over the row blocks i >= j of W_i L_ij, the upper part of the
// diagonal block left out.  (The sign does not matter to the squares taken of U.)
__global__ void __launch_bounds__(kRowsThreads)
rows_times_lower_kernel(const double* __restrict__ tiles, int ts, int nt, const double* __restrict__ W,
                        double* __restrict__ U, long long ldy) {
  extern __shared__ __align__(16) double sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const long long ts2 = (long long)ts * ts;
  const int j = blockIdx.x, nblk = gridDim.x, c0 = kStep * j, tj = c0 / ts, lc = c0 - tj * ts;
  auto fetch = [&](int i) {
    double* A = sm + 2 * ((i - j) & 1) * kStepBlock;
    const int r0 = kStep * i, ti = r0 / ts;
    load_block(A, W + r0 * ldy + kStep * blockIdx.y, ldy, kRowsThreads);
    load_block(A + kStepBlock, tiles + tile_slot(ti, tj, nt) * ts2 + (long long)lc * ts + (r0 - ti * ts), ts,
               kRowsThreads);
    cp_async_commit();
  };
  double c[8][4];
#pragma unroll
  for (int ni = 0; ni < 8; ++ni)
#pragma unroll
    for (int h = 0; h < 4; ++h) c[ni][h] = 0.0;
  fetch(j);
  for (int i = j; i < nblk; ++i) {
    if (i + 1 < nblk) {
      fetch(i + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    double* A = sm + 2 * ((i - j) & 1) * kStepBlock;
    double* B = A + kStepBlock;
    if (i == j) {
      for (int e = tid; e < kStep * kStep; e += kRowsThreads)
        if ((e & 63) < (e >> 6)) B[(e >> 6) * kStepLd + (e & 63)] = 0.0;
      __syncthreads();
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      double a[8];
      frag_a_neg(A, 16 * warp, 16 * kk, lane, a);
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        double b[4];
        frag_bt(B, 8 * ni, 16 * kk, lane, b);
        dmma_16816(c[ni], a, b);
      }
    }
    __syncthreads();
  }
  double* p = U + (long long)(c0 + 2 * t) * ldy + kStep * blockIdx.y + 16 * warp + 2 * g;
#pragma unroll
  for (int ni = 0; ni < 8; ++ni)
#pragma unroll
    for (int h = 0; h < 2; ++h) stg_v2f64(p + (8 * ni + h) * ldy, c[ni][h], c[ni][2 + h]);
}

// out[q * stride] = sum over the columns c < np of A(q, c) B(q, c): 32 rows x 8
// column groups per block, fixed order.
__global__ void __launch_bounds__(256)
rows_dot_kernel(const double* __restrict__ A, const double* __restrict__ B, long long ldy, int np, int m,
                double* __restrict__ out, int stride) {
  __shared__ double red[8][33];
  const int q = 32 * blockIdx.x + (threadIdx.x & 31), g = threadIdx.x >> 5;
  double acc = 0.0;
#pragma unroll 4
  for (int c = g; c < np; c += 8) acc = fma(A[c * ldy + q], B[c * ldy + q], acc);
  red[g][threadIdx.x & 31] = acc;
  __syncthreads();
  if (g != 0 || q >= m) return;
  double s = red[0][threadIdx.x];
  for (int i = 1; i < 8; ++i) s += red[i][threadIdx.x];
  out[(long long)q * stride] = s;
}

constexpr int rows_step_smem() { return (3 * kStepBlock + kStep) * (int)sizeof(double); }
constexpr int rows_times_smem() { return 4 * kStepBlock * (int)sizeof(double); }

// Column blocks per CTA of a step with nblk of them and `chunks` row chunks: a
// CTA's own solve costs about 1.25 block updates and two CTAs fit an SM, so the
// cheapest split has few partial waves (Fisher information N = 1,600, 75 chunks:
// 40.6 us a step on average, 47 with at most four blocks per CTA).
int rows_share(int nblk, int chunks) {
  const long long slots = 2LL * gemm_num_sms();
  int best = 1;
  double cost = 1e300;
  for (int share = 1; share <= 16 && share <= nblk; ++share) {
    const long long ctas = (long long)((nblk + share - 1) / share) * chunks;
    const double c = (double)((ctas + slots - 1) / slots) * (1.25 + share);
    if (c < cost) {
      cost = c;
      best = share;
    }
  }
  return best;
}

// blocks: the 64-column blocks that take part.
template <bool kBack>
int rows_solve(const double* tiles, int ts, int nt, int blocks, double* Y, double* X, long long ldy, int rows, int sym,
               cudaStream_t st) {
  static std::once_flag done[64];
  once_per_device(done, []() {
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(rows_step_kernel<false>, attr, rows_step_smem());
    cudaFuncSetAttribute(rows_step_kernel<true>, attr, rows_step_smem());
    cudaFuncSetAttribute(rows_times_lower_kernel, attr, rows_times_smem());
  });
  const int per = ts / kStep;
  for (int i = 0; i < blocks; ++i) {
    const int b = kBack ? blocks - 1 - i : i;
    const int nblk = kBack ? b : blocks - 1 - b;
    const int chunks = sym > 0 ? rows / kStep / sym * (nblk + 1) : rows / kStep;
    const int share = rows_share(sym > 0 ? (nblk + 1) / 2 : nblk, chunks);
    const dim3 grid(nblk > 0 ? (nblk + share - 1) / share : 1, chunks);
    const int k = b / per, kb = (b % per) * kStep;
    if (i == 0) {  // an ordinary launch: the factor and Y are complete
      rows_step_kernel<kBack><<<grid, kRowsThreads, rows_step_smem(), st>>>(tiles, ts, nt, k, kb, nblk, share, sym, Y,
                                                                            X, ldy);
      continue;
    }
    const int rc = launch_overlapped("rows_step_kernel", rows_step_kernel<kBack>, grid, dim3(kRowsThreads),
                                     rows_step_smem(), st, tiles, ts, nt, k, kb, nblk, share, sym, Y, X, ldy);
    if (rc != EGS_OK) return rc;
  }
  return launch_status("rows_step_kernel");
}

}  // namespace

// z := L^-1 z / L^-T z for the first `rows` rows of the nt x nt lower tiles; scratch
// holds 128 doubles.
int launch_vec_forward(const double* tiles, int ts, int nt, int rows, double* z, double* scratch, cudaStream_t st,
                       long long* launches) {
  return vec_solve<false>(tiles, ts, nt, rows, z, scratch, st, launches);
}
int launch_vec_backward(const double* tiles, int ts, int nt, int rows, double* z, double* scratch, cudaStream_t st,
                        long long* launches) {
  return vec_solve<true>(tiles, ts, nt, rows, z, scratch, st, launches);
}

// The same for `rows` (a multiple of 64) right-hand sides held as the rows of Y
// (column c of length ldy at Y + c ldy, 64 blocks columns): X := Y L^-T / Y L^-1 by the
// first `blocks` 64-column blocks of L.  Y is overwritten.
int launch_rows_forward(const double* tiles, int ts, int nt, int blocks, double* Y, double* X, long long ldy, int rows,
                        cudaStream_t st) {
  return rows_solve<false>(tiles, ts, nt, blocks, Y, X, ldy, rows, 0, st);
}
int launch_rows_backward(const double* tiles, int ts, int nt, int blocks, double* Y, double* X, long long ldy,
                         int rows, cudaStream_t st) {
  return rows_solve<true>(tiles, ts, nt, blocks, Y, X, ldy, rows, 0, st);
}

// X := Y L^-T for `count` stacked square matrices whose results are symmetric: only the
// 64 x 64 blocks on and below each diagonal are computed, a third of the work.
int launch_rows_forward_symmetric(const double* tiles, int ts, int nt, int blocks, double* Y, double* X, int count,
                                  cudaStream_t st) {
  const int rows = count * blocks * kStep;
  return rows_solve<false>(tiles, ts, nt, blocks, Y, X, rows, rows, blocks, st);
}

// U := -W L for the lower tiles (after a launch_rows_* call of this process on the device).
int launch_rows_times_lower(const double* tiles, int ts, int nt, int blocks, const double* W, double* U, long long ldy,
                            int rows, cudaStream_t st) {
  rows_times_lower_kernel<<<dim3(blocks, rows / kStep), kRowsThreads, rows_times_smem(), st>>>(tiles, ts, nt, W, U,
                                                                                            ldy);
  return launch_status("rows_times_lower_kernel");
}

// out[q * stride] = (row q of A) . (row q of B) for q < m, np columns.
void launch_rows_dot(const double* A, const double* B, long long ldy, int np, int m, double* out, int stride,
                     cudaStream_t st) {
  rows_dot_kernel<<<(m + 31) / 32, 256, 0, st>>>(A, B, ldy, np, m, out, stride);
}

}  // namespace egs
