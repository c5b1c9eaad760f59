// One 64-column step of the panel factorisation of a tall tile column: the
// device body shared by the single-problem kernel (potrf.cu) and the batched
// kernel (batch.cu).
//
// A step factors the 64 x 64 diagonal block, solves every row below it and
// applies the 64 new columns to the columns right of it inside the same outer
// block, in ONE launch: one CTA per 64-row chunk below the block.  Every CTA
// factors the diagonal block itself and solves the other row chunk whose solved
// rows its update needs, so no CTA waits for another one.  It is bound by the
// chain of 64 dependent pivots, not by work: three dependent launches for the
// three parts took 58-70 us per step whatever the panel's height, a step now
// takes 13 to 17 us while every chunk has an SM, 17 to 30 above (N = 1,600, tile 320:
// panels 1.46 -> 0.44 ms per evaluation, the forward solve below 0.51 -> 0; N = 10,000,
// tile 960: 11.5 -> 5.0 and 6.9 -> 0).
// The redundant arithmetic runs on SMs that would otherwise be idle.
// Outer blocks are two 64-column blocks wide: wider ones make every CTA solve
// more foreign chunks (each costs as much FP64 time as its own), narrower ones
// leave more to the K = 64 update launches (N = 1,600 / N = 20,011 mixed / 512-problem
// batch: one block 533 us / 32.6 ms / 83.7 ms, two 556 / 31.7 / 78.3, three 583 /
// 32.0 / 86.0).
//
// The pivots run in one warp, eight at a time in registers: every lane holds
// the 8 x 8 block, so no pivot waits for an exchange between lanes (16 columns
// with shuffles took 4,900 cycles per 16 pivots, this form 2 x 1,400 alone).  The other
// warps solve their rows against the previous 16 columns meanwhile (two warps
// per 64-row chunk, one thread per row for the 16-column substitution, DMMA for
// the rest), so only the last 16 columns of the row solve and the DMMA update
// follow the last pivot.
//
// Rows below the outer block are read and written by their own CTA only.  The
// diagonal block and the rows inside the outer block are read by every CTA, so
// their solved values go to a scratch slot instead, and the next step's launch
// (or panel_flush_kernel after the last one) copies them to their place: two
// slots, used alternately.
//
// The observation vector rides along: z_k := L_kk^-1 z_k is solved like one more
// row, and every row chunk applies z_i -= L_ik z_k from the solved rows it has
// in shared memory, so the factorisation ends with Z = L^-1 Z and reads no part
// of L again for it.
#pragma once
#include "common.cuh"
#include "dmma.cuh"

namespace egs {

constexpr int kStep = 64;           // columns of a step, rows of a chunk
constexpr int kStepLd = 68;         // shared-memory column stride: fragment loads hit distinct banks;
                                    // the padding of the diagonal block's columns holds the pivots
constexpr int kStepBlock = kStep * kStepLd;
constexpr int kStepMaxBlocks = 2;   // most 64-column blocks of an outer block
constexpr int kStepThreads = 128 * ((2 * kStepMaxBlocks + 4) / 3);
constexpr int kStepHelpers = 3 * kStepThreads / 128;  // warps beside the pivot warp's sub-partition
static_assert(2 * kStepMaxBlocks + 2 <= kStepHelpers, "two warps per row chunk and two for the diagonal block");
constexpr int kScratchLd = kStepMaxBlocks * kStep;
constexpr int kScratchSlot = kScratchLd * kStep + kStep;  // solved rows, then z_k
constexpr int kScratchDoubles = 2 * kScratchSlot;

// Further 64-column blocks (0 or 1) in the outer block of column kb of a tile
// with cols columns: outer blocks are pairs, the last one may be a single block.
__host__ __device__ constexpr int panel_outer_rest(int cols, int kb) {
  return ((kb / kStep) & 1) == 0 && kb + kStep < cols ? 1 : 0;
}
static_assert(kStepMaxBlocks == 2, "panel_outer_rest pairs the blocks");

// Dynamic shared memory of a step with nb further blocks in its outer block:
// the diagonal block, the CTA's rows, nb other row chunks, 1/L_jj and z_k.
__host__ __device__ constexpr int panel_step_smem(int nb) {
  return ((2 + nb) * kStepBlock + 2 * kStep) * (int)sizeof(double);
}

__device__ __forceinline__ void cp_async16(double* dst, const double* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A fragment (16 rows x 16 k) of the column-major block x (rows row0 + 2g and
// row0 + 2g + 1 are MMA rows g and g + 8), negated.
__device__ __forceinline__ void frag_a_neg(const double* x, int row0, int k0, int lane, double (&a)[8]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double2 v = *reinterpret_cast<const double2*>(x + (k0 + t + 4 * j) * kStepLd + row0 + 2 * g);
    a[2 * j] = -v.x;
    a[2 * j + 1] = -v.y;
  }
}
// B fragment (8 columns x 16 k): column n is row n0 + n of the block x.
__device__ __forceinline__ void frag_b(const double* x, int n0, int k0, int lane, double (&b)[4]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) b[i] = x[(k0 + t + 4 * i) * kStepLd + n0 + g];
}
// C fragment (16 rows x 8 columns) at (row0, n0) of the block x.
__device__ __forceinline__ void frag_c_load(const double* x, int row0, int n0, int lane, double (&c)[4]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double2 v = *reinterpret_cast<const double2*>(x + (n0 + 2 * t + h) * kStepLd + row0 + 2 * g);
    c[h] = v.x;
    c[2 + h] = v.y;
  }
}
__device__ __forceinline__ void frag_c_store(double* x, int row0, int n0, int lane, const double (&c)[4]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h)
    *reinterpret_cast<double2*>(x + (n0 + 2 * t + h) * kStepLd + row0 + 2 * g) = make_double2(c[h], c[2 + h]);
}

// x(rows row0 .. row0+15, columns n0 .. n0+15) -= A B^T with A a negated
// fragment and B the rows n0 .. n0+15 of block d at columns k0 .. k0+15.
template <int MB>
__device__ __forceinline__ void block_update_16(double* x, int row0, int n0, const double* d, int k0, int lane,
                                                const double (&a)[MB][8]) {
  double c[MB][2][4], b[2][4];
  frag_b(d, n0, k0, lane, b[0]);
  frag_b(d, n0 + 8, k0, lane, b[1]);
#pragma unroll
  for (int m = 0; m < MB; ++m) {
    frag_c_load(x, row0 + 16 * m, n0, lane, c[m][0]);
    frag_c_load(x, row0 + 16 * m, n0 + 8, lane, c[m][1]);
  }
#pragma unroll
  for (int m = 0; m < MB; ++m) {
    dmma_16816(c[m][0], a[m], b[0]);
    dmma_16816(c[m][1], a[m], b[1]);
  }
#pragma unroll
  for (int m = 0; m < MB; ++m) {
    frag_c_store(x, row0 + 16 * m, n0, lane, c[m][0]);
    frag_c_store(x, row0 + 16 * m, n0 + 8, lane, c[m][1]);
  }
}

// 1 / sqrt(d) for normal d well inside the exponent range: the hardware's
// approximation y (about 2^-20) and one step of Householder's third-order
// iteration on its residual e, y (1 + e / 2 + 3 e^2 / 8).  The omitted 5 e^3 / 16 is
// below 2^-58, the rounding of d y in e puts 2^-54 into the result, its own rounding
// 2^-53: within 2^-52 of the root's reciprocal, as a rounded root and a rounded division are.
// A shorter dependent chain than rsqrt(), which the pivots below wait for.
__device__ __forceinline__ double step_rsqrt(double d) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-(d * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// Cholesky of the 8 x 8 lower block l in registers, every lane the same values:
// no exchange between lanes, so the chain per pivot is rsqrt, scale and one
// fused multiply-add.  l[j][j] becomes 1 / L_jj.  Returns a mask of the pivots outside
// the range of the fast rsqrt (zero, negative, NaN, subnormal, huge); kSafe uses
// rsqrt() and returns the mask of pivots that are not positive (or NaN).
// The pivots themselves go to piv (stride kStepLd), for step_roots.
template <bool kSafe>
__device__ __forceinline__ unsigned step_factor8(double (&l)[8][8], double* piv, int lane) {
  unsigned mask = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const double d = l[j][j];
    if (lane == 0) piv[j * kStepLd] = d;
    if constexpr (kSafe) {
      if (!(d > 0.0)) mask |= 1u << j;
      l[j][j] = rsqrt(d);
    } else {
      // exponent field in [0x05d, 0x79d): about 1e-280 .. 1e+280, sign bit clear
      if ((unsigned)__double2hiint(d) - 0x05d00000u >= 0x74000000u) mask |= 1u << j;
      l[j][j] = step_rsqrt(d);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i > j) l[i][j] *= l[j][j];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c > j && i >= c) l[i][c] = fma(-l[i][j], l[c][j], l[i][c]);
  }
  return mask;
}

// y := y L^-T for one row of 8 values (l[j][j] = 1 / L_jj).
__device__ __forceinline__ void step_subst8(double (&y)[8], const double (&l)[8][8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    y[j] *= l[j][j];
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (c > j) y[c] = fma(-y[j], l[c][j], y[c]);
  }
}

// y -= x L^T with L the rows n0 .. n0+7 of D at columns k0 .. k0+7.
__device__ __forceinline__ void step_update8(double (&y)[8], const double (&x)[8], const double* D, int n0, int k0) {
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int n = 0; n < 8; n += 2) {
      const double2 v = *reinterpret_cast<const double2*>(D + (k0 + q) * kStepLd + n0 + n);
      y[n] = fma(-x[q], v.x, y[n]);
      y[n + 1] = fma(-x[q], v.y, y[n + 1]);
    }
}

__device__ __forceinline__ void step_load8(double (&y)[8], const double* p) {
#pragma unroll
  for (int c = 0; c < 8; ++c) y[c] = p[c * kStepLd];
}
__device__ __forceinline__ void step_store8(double* p, const double (&y)[8]) {
#pragma unroll
  for (int c = 0; c < 8; ++c) p[c * kStepLd] = y[c];
}

// One warp: columns 8 b .. 8 b + 7 of the diagonal block D, rows 8 b .. 63: the
// update with the previous eight columns (older ones are already in), the 8 x 8
// Cholesky and the solve of the rows.  Lane r holds rows r and r + 32; finished
// rows compute values of the unused upper part.  pinv receives 1 / L_jj.
__device__ __forceinline__ void step_pivots8(double* D, double* pinv, int b, int gcol, int* info, int lane) {
  double* col = D + (8 * b) * kStepLd;
  const double* prev = col - 8 * kStepLd;
  const int hi = b < 4 ? 0 : 32;  // the half that holds the block's own rows
  double y[8];
  if (b > 0) {
    double x[8];
    step_load8(y, col + hi + lane);
    step_load8(x, prev + hi + lane);
    step_update8(y, x, D, 8 * b, 8 * (b - 1));
    step_store8(col + hi + lane, y);
    __syncwarp();
  }
  double l[8][8];
  auto load_block = [&]() {
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int i = 0; i < 8; i += 2)
        if (i + 1 >= c) {
          const double2 v = *reinterpret_cast<const double2*>(col + c * kStepLd + 8 * b + i);
          if (i >= c) l[i][c] = v.x;
          l[i + 1][c] = v.y;
        }
  };
  load_block();
  if (step_factor8<false>(l, col + kStep, lane)) {
    load_block();
    const unsigned bad = step_factor8<true>(l, col + kStep, lane);
    if (bad && info && lane == 0) atomicCAS(info, 0, gcol + 8 * b + __ffs(bad));
  }
  step_load8(y, col + hi + lane);  // not kept across the pivots: registers are short
  step_subst8(y, l);
  __syncwarp();
  step_store8(col + hi + lane, y);
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) pinv[8 * b + j] = l[j][j];
  }
  if (b < 4) {
    // the other half against L and 1 / L_jj in shared memory (registers are short)
    step_load8(y, col + 32 + lane);
    if (b > 0) {
      double x[8];
      step_load8(x, prev + 32 + lane);
      step_update8(y, x, D, 8 * b, 8 * (b - 1));
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      y[j] *= pinv[8 * b + j];
#pragma unroll
      for (int c = 0; c < 8; c += 2)
        if (c + 1 > j) {
          const double2 v = *reinterpret_cast<const double2*>(col + j * kStepLd + 8 * b + c);
          if (c > j) y[c] = fma(-y[j], v.x, y[c]);
          y[c + 1] = fma(-y[j], v.y, y[c + 1]);
        }
    }
    step_store8(col + 32 + lane, y);
  }
}

// One warp: L_jj, the rounded root of pivot j, which waits in the padding of column j.
// The substitutions use 1 / L_jj, so the root is off the pivots' chain (pivot times
// reciprocal, without this, is up to one unit in the last place further off).
__device__ __forceinline__ void step_roots(double* D, int lane) {
  for (int j = lane; j < kStep; j += 32) D[j * kStepLd + j] = sqrt(D[j * kStepLd + kStep]);
}

// The rank-8 update of the diagonal block's columns from 8 (b + 1) on with the
// columns 8 (b - 1) .. 8 b - 1, by warp `w` of `nw`: 16 x 8 tiles on and below
// the diagonal.
__device__ __forceinline__ void step_trailing8(double* D, int b, int w, int nw, int lane) {
  const int g = lane >> 2, t = lane & 3, k0 = 8 * (b - 1);
  int idx = 0;
#pragma unroll 1
  for (int j = b + 1; j < 8; ++j)
#pragma unroll 1
    for (int m = j >> 1; m < 4; ++m, ++idx) {
      if (idx % nw != w) continue;
      double a[4], bb[2], c[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double2 v = *reinterpret_cast<const double2*>(D + (k0 + t + 4 * i) * kStepLd + 16 * m + 2 * g);
        a[2 * i] = -v.x;
        a[2 * i + 1] = -v.y;
        bb[i] = D[(k0 + t + 4 * i) * kStepLd + 8 * j + g];
      }
      frag_c_load(D, 16 * m, 8 * j, lane, c);
      dmma_1688(c, a, bb);
      frag_c_store(D, 16 * m, 8 * j, lane, c);
    }
}

// v := v L_ss^-T for one row of 16 values (right-looking substitution); L_ss is
// the 16 x 16 block at `blk` (column stride kStepLd).
__device__ __forceinline__ void step_subst16(double (&v)[16], const double* blk, const double* pinv) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    v[j] *= pinv[j];
    const double xj = v[j];
    if (j + 1 < 16 && ((j + 1) & 1)) v[j + 1] = fma(-xj, blk[j * kStepLd + j + 1], v[j + 1]);
#pragma unroll
    for (int c = (j + 2) & ~1; c < 16; c += 2) {
      const double2 l2 = *reinterpret_cast<const double2*>(blk + j * kStepLd + c);
      v[c] = fma(-xj, l2.x, v[c]);
      v[c + 1] = fma(-xj, l2.y, v[c + 1]);
    }
  }
}

// One warp: rows row0 .. row0 + 16 MB - 1 of block X (MB = 1: the upper lanes
// repeat the lower ones), sub-block q: substitution against L_qq, then the update
// of the later sub-blocks.
template <int MB>
__device__ __forceinline__ void step_rows(double* X, const double* D, const double* pinv, int q, int row0, int lane) {
  double* xr = X + row0 + (MB == 2 ? lane : lane & 15);
  {
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = xr[(16 * q + j) * kStepLd];
    step_subst16(v, D + (16 * q) * kStepLd + 16 * q, pinv + 16 * q);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 16; ++j) xr[(16 * q + j) * kStepLd] = v[j];
  }
  __syncwarp();
  if (q == 3) return;
  double a[MB][8];
#pragma unroll
  for (int m = 0; m < MB; ++m) frag_a_neg(X, row0 + 16 * m, 16 * q, lane, a[m]);
#pragma unroll 1
  for (int n0 = 16 * (q + 1); n0 < kStep; n0 += 16) block_update_16<MB>(X, row0, n0, D, 16 * q, lane, a);
  __syncwarp();
}

// This lane's elements of a 16 x 32 warp tile of C (column stride ts).
__device__ __forceinline__ void step_load_c(const double* p, int ts, double (&cv)[4][4]) {
#pragma unroll
  for (int ni = 0; ni < 4; ++ni)
#pragma unroll
    for (int h = 0; h < 2; ++h) ldg_v2f64(p + (long long)(8 * ni + h) * ts, cv[ni][h], cv[ni][2 + h]);
}

// Barrier of the whole block, callable from different branches, and of the pivot
// and diagonal-block warps only.
__device__ __forceinline__ void bar_sync_all() { asm volatile("bar.sync 0;" ::: "memory"); }
__device__ __forceinline__ void bar_sync_diag() { asm volatile("bar.sync 1, 96;" ::: "memory"); }

// The whole step for row chunk `chunk` (-1: no rows below the block).  col is
// tile (k, k) of a column of contiguous ts x ts tiles, kb the block's first
// column in it, nb the number of further 64-column blocks of its outer block;
// z (may be null) the vector's segment of tile row k; out the scratch slot.
// Dynamic shared memory: panel_step_smem(nb).
__device__ __forceinline__ void panel_step_body(double* __restrict__ sm, double* col, int ts, int chunk, int kb, int nb,
                                                int gcol, int* info, double* z, double* __restrict__ out) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* D = sm;
  double* A = sm + kStepBlock;
  double* pinv = sm + (2 + nb) * kStepBlock;
  double* zk = pinv + kStep;
  const bool inner = chunk >= 0 && chunk < nb;        // own rows lie inside the outer block
  const int nother = chunk < 0 ? 0 : min(chunk, nb);  // other chunks this CTA solves
  const int ncol = chunk < 0 ? 0 : min(chunk + 1, nb);
  const int nrc = chunk < 0 ? 0 : 1 + nother;
  const long long ts2 = (long long)ts * ts;
  const int g = kb + kStep + kStep * chunk;  // own first row, from row 0 of tile row k
  double* own = col;
  if (chunk >= 0) own = col + (g / ts) * ts2 + (g % ts);  // column 0 of the own rows

  for (int e = tid; e < kStep * kStep / 2; e += kStepThreads) {
    const int c = e >> 5, r = 2 * (e & 31);
    cp_async16(D + c * kStepLd + r, col + (long long)(kb + c) * ts + kb + r);
  }
  cp_async_commit();
  if (z && tid < kStep) zk[tid] = z[kb + tid];
  // the rows' part of z, subtracted from at the end by the last two warps
  const int zr = tid - (kStepThreads - kStep);
  const double zi = (z && chunk >= 0 && zr >= 0) ? z[g + zr] : 0.0;
  cp_async_wait<0>();
  __syncthreads();
  // the pivots start; the row blocks, needed two rounds later, arrive beside them
  if (warp != 0) {
    for (int b = 0; b < nrc; ++b) {
      const double* src = (b == 0) ? own : col + kb + kStep * b;
      double* dst = A + b * kStepBlock;
      for (int e = tid - 32; e < kStep * kStep / 2; e += kStepThreads - 32) {
        const int c = e >> 5, r = 2 * (e & 31);
        cp_async16(dst + c * kStepLd + r, src + (long long)(kb + c) * ts + r);
      }
    }
    cp_async_commit();
  }

  // Warp 0 runs the pivots and has its SM sub-partition to itself (an FP64 MMA
  // of another warp would hold up its chain); warps 1-3 (mod 4) are helpers:
  // 0 .. 2 nrc - 1 solve rows, the last two update the diagonal block, the very
  // last also solves z.
  const int helper = (warp & 3) ? (warp >> 2) * 3 + (warp & 3) - 1 : -1;
  const int rc = helper >> 1, half = helper & 1;
  const bool rows_warp = helper >= 0 && helper < 2 * nrc;
  const int diag_warp = helper - (kStepHelpers - 2);  // 0, 1: diagonal-block warps
  // z_k like one more row: 16 columns by substitution (one lane), the rest by the warp
  auto z_substep = [&](int q) {
    if (!z) return;
    if (lane == 0) {
      double v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = zk[16 * q + j];
      step_subst16(v, D + (16 * q) * kStepLd + 16 * q, pinv + 16 * q);
#pragma unroll
      for (int j = 0; j < 16; ++j) zk[16 * q + j] = v[j];
    }
    __syncwarp();
    for (int r = 16 * (q + 1) + lane; r < kStep; r += 32) {
      double acc = zk[r];
#pragma unroll
      for (int j = 0; j < 16; ++j) acc = fma(-D[(16 * q + j) * kStepLd + r], zk[16 * q + j], acc);
      zk[r] = acc;
    }
    __syncwarp();
  };
  // Eight rounds of eight pivots.  The pivot and diagonal-block warps meet after
  // every round; everyone after every second one, when 16 more columns of L are
  // final for the row solves.
  if (warp == 0) {
#pragma unroll 1
    for (int b = 0; b < 8; ++b) {
      step_pivots8(D, pinv, b, gcol, info, lane);
      if (b & 1) {
        cp_async_wait<0>();
        bar_sync_all();
      } else {
        bar_sync_diag();
      }
    }
  } else if (diag_warp >= 0) {
#pragma unroll 1
    for (int b = 0; b < 8; ++b) {
      if (b > 0) step_trailing8(D, b, diag_warp, 2, lane);
      if (diag_warp == 1 && b >= 2 && !(b & 1)) z_substep((b >> 1) - 1);
      if (b & 1) {
        cp_async_wait<0>();
        bar_sync_all();
      } else {
        bar_sync_diag();
      }
    }
  } else {
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
      if (s > 0 && rows_warp) step_rows<2>(A + rc * kStepBlock, D, pinv, s - 1, 32 * half, lane);
      cp_async_wait<0>();
      bar_sync_all();
    }
  }
  // C of this warp's first update tile, in flight during the last row sub-step
  const int gq = lane >> 2, tq = lane & 3;
  // warp tile -> its first element for this lane: column block tile / 8, 16 rows, 32 columns
  auto tile_ptr = [&](int tile) {
    const int c = tile >> 3, mb = (tile >> 1) & 3, n2 = tile & 1;
    return own + (long long)(kb + kStep + kStep * c + 32 * n2 + 2 * tq) * ts + 16 * mb + 2 * gq;
  };
  const int ntiles = 8 * ncol;
  double cv[4][4];
  if (warp < ntiles) step_load_c(tile_ptr(warp), ts, cv);
  if (rows_warp) step_rows<2>(A + rc * kStepBlock, D, pinv, 3, 32 * half, lane);
  if (diag_warp == 0) step_roots(D, lane);
  if (diag_warp == 1) z_substep(3);
  __syncthreads();

  grid_dependents_launch();
  // solved rows out
  if (chunk >= 0) {
    double* dst = inner ? out + kStep * (chunk + 1) : own + (long long)kb * ts;
    const long long ld = inner ? kScratchLd : ts;
    for (int e = tid; e < kStep * kStep / 2; e += kStepThreads) {
      const int c = e >> 5, r = 2 * (e & 31);
      *reinterpret_cast<double2*>(dst + c * ld + r) = *reinterpret_cast<const double2*>(A + c * kStepLd + r);
    }
  }
  if (chunk <= 0) {
    for (int e = tid; e < kStep * kStep / 2; e += kStepThreads) {
      const int c = e >> 5, r = 2 * (e & 31);
      *reinterpret_cast<double2*>(out + c * kScratchLd + r) = *reinterpret_cast<const double2*>(D + c * kStepLd + r);
    }
    if (z && tid < kStep) out[kScratchLd * kStep + tid] = zk[tid];
  }
  if (z && chunk >= 0 && zr >= 0) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll 4
    for (int c = 0; c < kStep; c += 4) {
      s0 = fma(A[c * kStepLd + zr], zk[c], s0);
      s1 = fma(A[(c + 1) * kStepLd + zr], zk[c + 1], s1);
      s2 = fma(A[(c + 2) * kStepLd + zr], zk[c + 2], s2);
      s3 = fma(A[(c + 3) * kStepLd + zr], zk[c + 3], s3);
    }
    z[g + zr] = zi - ((s0 + s1) + (s2 + s3));
  }
  // update of the later columns of the outer block: 16 x 32 warp tiles, K = 64
#pragma unroll 1
  for (int tile = warp; tile < ntiles; tile += kStepThreads / 32) {
    if (tile != warp) step_load_c(tile_ptr(tile), ts, cv);
    const int c = tile >> 3, mb = (tile >> 1) & 3, n2 = tile & 1;
    const double* B = (inner && c == chunk) ? A : A + (c + 1) * kStepBlock;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      double a[8];
      frag_a_neg(A, 16 * mb, 16 * kk, lane, a);
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        double b[4];
        frag_b(B, 32 * n2 + 8 * ni, 16 * kk, lane, b);
        dmma_16816(cv[ni], a, b);
      }
    }
    double* p = tile_ptr(tile);
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) stg_v2f64(p + (long long)(8 * ni + h) * ts, cv[ni][h], cv[ni][2 + h]);
  }
}

// Rows 64 f .. 64 f + 63 of a scratch slot to their place: the lower part of the
// diagonal block (f = 0) or a solved row chunk of the outer block.
__device__ __forceinline__ void panel_flush_body(const double* __restrict__ slot, double* __restrict__ col, int ts,
                                                 int kb, int f, double* __restrict__ z) {
  for (int e = threadIdx.x; e < kStep * kStep / 2; e += blockDim.x) {
    const int c = e >> 5, r = 2 * (e & 31);
    const double2 v = *reinterpret_cast<const double2*>(slot + c * kScratchLd + kStep * f + r);
    double* dst = col + (long long)(kb + c) * ts + kb + kStep * f + r;
    if (f > 0 || r >= c) {
      *reinterpret_cast<double2*>(dst) = v;
    } else if (r + 1 >= c) {
      dst[1] = v.y;
    }
  }
  if (f == 0 && z && threadIdx.x < kStep) z[kb + threadIdx.x] = slot[kScratchLd * kStep + threadIdx.x];
}

}  // namespace egs
