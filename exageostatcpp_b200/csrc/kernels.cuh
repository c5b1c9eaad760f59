// Launch helpers shared by the translation units of the B200 path.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include "common.cuh"
#include "bessel_k.cuh"

namespace egs {

// Stream-ordered device memory from the library's pool (capi.cu); released with cudaFreeAsync.
int alloc_from_pool(void** p, size_t bytes, cudaStream_t st);

int make_matern_params(const double* theta, MaternParams* out);
// Builds the polynomial table of K_nu for theta (ktab: kKtabDoubles device
// doubles), then generates every lower tile.
int launch_matern_tiles(double* tiles, const double* x, const double* y, int n, int ts, int nt,
                        const MaternParams* dparams, double* ktab, cudaStream_t st);
// Polynomial tables of nproblems parameter sets (tab: nproblems * kKtabDoubles).
void launch_matern_ktab(const MaternParams* params, double* tab, int nproblems, cudaStream_t st);
int launch_matern_block(double* a, int lda, int rows, int cols, const double* x1, const double* y1,
                        const double* x2, const double* y2, const MaternParams& p, cudaStream_t st);
// The same with theta's parameters and table already on the device (launch_matern_ktab).
int launch_matern_block_tab(double* a, int lda, int rows, int cols, const double* x1, const double* y1,
                            const double* x2, const double* y2, const MaternParams* params, const double* ktab,
                            cudaStream_t st);

// Factorisation building blocks (potrf.cu).  All offsets are element offsets
// inside a tile; tiles are addressed by lower-tile slot.
// Panel steps of one factorisation (panel_step.cuh): the scratch slots the steps
// use alternately, and the step whose solved rows are still in its slot.
struct PanelChain {
  double* scratch = nullptr;  // panel_scratch_doubles()
  int parity = 0;             // slot of the next step
  int chunks = 0;             // 64-row chunks of the last step still in the other slot (0: none)
  double* col = nullptr;
  int kb = 0, ts = 0;
  double* z = nullptr;
};
long long panel_scratch_doubles();
// Rows (and columns) of a problem of n points that take part in factorisations and
// solves: the 64-row blocks with a real row.  The padding beyond them is the
// identity and stays it.
__host__ __device__ inline int factor_rows(int n) { return (n + 63) / 64 * 64; }
// One step: col is tile (k, k) of a contiguous tile column, rows_below the rows
// under the 64 x 64 block at (kb, kb), nb the further 64-column blocks of its
// outer block (updated by the step), gcol the global column of the block (for
// info), z (or null) the segment of tile row k of a vector that becomes L^-1 z.
// The diagonal block, z's segment and the solved rows inside the outer block
// reach their place with the next step's launch or launch_panel_flush.
int launch_panel_step(double* col, int ts, int rows_below, int kb, int nb, int gcol, int* info, double* z,
                      PanelChain& ch, cudaStream_t st);
int launch_panel_flush(PanelChain& ch, cudaStream_t st);
// Triangular solves against a finished factor (solve.cu): one vector in place
// of `rows` entries (a multiple of 64; scratch: 128 doubles), or the rows of a matrix.
int launch_vec_forward(const double* tiles, int ts, int nt, int rows, double* z, double* scratch, cudaStream_t st,
                       long long* launches);
int launch_vec_backward(const double* tiles, int ts, int nt, int rows, double* z, double* scratch, cudaStream_t st,
                        long long* launches);
int launch_rows_forward(const double* tiles, int ts, int nt, int blocks, double* Y, double* X, long long ldy, int rows,
                        cudaStream_t st);
int launch_rows_backward(const double* tiles, int ts, int nt, int blocks, double* Y, double* X, long long ldy,
                         int rows, cudaStream_t st);
int launch_rows_forward_symmetric(const double* tiles, int ts, int nt, int blocks, double* Y, double* X, int count,
                                  cudaStream_t st);
int launch_rows_times_lower(const double* tiles, int ts, int nt, int blocks, const double* W, double* U, long long ldy,
                            int rows, cudaStream_t st);
void launch_rows_dot(const double* A, const double* B, long long ldy, int np, int m, double* out, int stride,
                     cudaStream_t st);
int launch_logdet_partials(const double* tiles, int ts, int nt, int n, double* partial, cudaStream_t st);
int launch_finalize(const double* partial, int nt, const double* z, int n, double* result, const int* info,
                    cudaStream_t st);
void launch_sumsq_diff(const double* a, const double* b, int n, double* out, cudaStream_t st);
void launch_trmv(const double* tiles, int ts, int nt, const double* e, double* part, double* z, cudaStream_t st);
void launch_gemv_t_block(const double* a, long long lda, int rows, int cols, const double* w, double* out,
                         cudaStream_t st);

// Band (diagonal super-tile) factorisation on logical tiles of dts elements,
// element by element inside the lower-tile pool (dst.cu); for dts != ts.
int launch_dst_band(double* tiles, int ts, int nt, int n, int dts, int band, int* info, cudaStream_t st);

// FP64 tensor-core update C -= A * B^T over global row indices (dgemm_tma.cu).
// Every operand row is a global row of one problem (tile row g / ts); A and B take
// their K columns from one tile column starting at a local column offset; C is
// addressed by (global row, global column), upper tiles never written.
struct GemmDesc {
  int M, N, K;
  int a_row0, a_col0, a_tcol;
  int b_row0, b_col0, b_tcol;
  int c_row0, c_col0;
  int lower;
  int MB, NB;
  long long total;
  int ts, nt, np;
  long long tile_base;  // slot of this problem's tile (0, 0) in a pool of problems
  // C addressing: c_mode 0 = lower-tile pool (tile_base + tile_slot(ti, tj, nt));
  // c_mode 1 = FP64 band pool of a mixed-precision problem: only tiles with
  // ti - tj <= c_band are written, at slot (c_tile_off + tj) * (c_band + 1) + (ti - tj);
  // c_mode 2 = lower-tile pool, only tiles with ti - tj <= c_band.
  int c_mode, c_band, c_tile_off;
  int cfg;  // tile shape of the launch (dgemm_tma.cu); set before finish_desc
};

// Batched launches: blocks [begin[j], begin[j+1]) belong to job j.
struct GemmJobs {
  const GemmDesc* jobs;
  const long long* begin;
  int njobs;
  long long total;
};

void finish_desc(GemmDesc& d);  // fills MB, NB, total
int gemm_tile_shape(long long total);  // cfg of a launch of `total` blocks of shape 0
int launch_gemm_batched(const void* tmap, double* tiles, int cfg, const GemmDesc* jobs, const long long* begin,
                        int njobs, long long total, int* err, cudaStream_t st);
int gemm_init_tensor_map(void* tmap_storage, double* tiles, int ts, long long ntiles);
// The driver's cuTensorMapEncodeTiled (looked up once).
int tensor_map_encoder(void** fn);
int launch_gemm_trailing(const void* tmap, double* tiles, int ts, int nt, int rows, int k, int* err, cudaStream_t st);
int launch_gemm_band(const void* tmap, double* tiles, int ts, int nt, int rows, int k, int band, int* err,
                     cudaStream_t st);
int launch_gemm_rows(const void* tmap, double* tiles, int ts, int nt, int M, int N, int K, int a_row0,
                     int a_col0, int a_tcol, int b_row0, int b_col0, int b_tcol, int c_row0, int c_col0,
                     int lower, int* err, cudaStream_t st);
int gemm_num_sms();

// Mixed-precision evaluation (mixed.cu, split_gemm.cu).
void launch_matern_mixed(double* band, float* off, const double* x, const double* y, int n, int ts,
                         const int4* tinfo, long long ntiles, const MaternParams* params, double* ktab,
                         cudaStream_t st);
void launch_gather_column(const double* band, const float* off, double* W, int ts, int nt, int b, int k,
                          cudaStream_t st);
void launch_scatter_column(const double* W, double* band, float* off, double* inv, int ts, int nt, int b, int k,
                           cudaStream_t st);
void launch_logdet_band(const double* band, int ts, int nt, int b, int n, double* partial, cudaStream_t st);
void launch_mixed_solve(const double* band, const float* off, const double* inv, int ts, int nt, int b, double* v,
                        double* tmp, cudaStream_t st, long long* launches);
void launch_gather_panel(const double* band, double* W2, int ts, int b, int nb, int k, cudaStream_t st);
void launch_scatter_panel(const double* W2, double* band, double* inv, double* W, int ts, int b, int nb, int k,
                          cudaStream_t st);
void launch_scatter_offband(const double* W, float* off, int ts, int nt, int b, int nb, int k, cudaStream_t st);
const float* offband_tile(const float* off, int ts, int nt, int b, int i, int k);
long long residual_scratch_doubles(int n);
void launch_add_inplace(double* a, const double* b, int n, cudaStream_t st);
void launch_matern_residual(const double* x, const double* y, const double* z, const double* v, int n, int np,
                            const MaternParams* params, const double* ktab, double* scratch, double* r,
                            cudaStream_t st);
void launch_finalize_mixed(const double* partial, int nt, const double* z, const double* v, const double* w, int n,
                           double* result, const int* info, cudaStream_t st);
int split_tensor_map(void* storage, const __half* base, int ts, long long rows);
int split_c_map(void* tm_c, const float* c_pool, int ts, long long nslots);
void launch_panel_split(const double* W, int ts, int t0, int ntiles, int row_tile0, float* inv_scale, __half* Ph,
                        __half* Pl, cudaStream_t st);
long long split_targets(int nt, int band, int k);
int ozaki_slices();
int ozaki_tensor_map(void* storage, const int8_t* slices, int ts, long long rows);
int launch_ozaki_slice(const double* W, int ts, int t0, int ntiles, int row_tile0, double* scale, int8_t* slices,
                        long long rows, cudaStream_t st);
}  // namespace egs
#include <vector>
namespace egs {
long long ozaki_targets(int ts, int nt, int band, int k, std::vector<int4>& out);
long long ozaki_trsm_targets(int ts, int nt, int first, std::vector<int4>& out);
int launch_panel_prepare(const double* W, int ts, int t0, int ntiles, int row_tile0, double* oz_scale,
                          int8_t* slices, long long rows, float* inv_scale, __half* Ph, __half* Pl, cudaStream_t st);
int launch_ozaki_slice_f32(const float* tiles0, int ts, int ntiles, int row_tile0, double* scale, int8_t* slices,
                            long long rows, cudaStream_t st);
void launch_ozaki_slice_rows(const double* src, int ts, long long row0, double* scale, int8_t* slices,
                             long long rows, cudaStream_t st);
int launch_ozaki_trsm(const void* tm_s, const int4* targets, int ntargets, long long total, int ts, int k,
                      long long b_row_base, double* w_out, const double* scale, int* err, cudaStream_t st);
int launch_ozaki_band(const void* tm_s, const int4* targets, int ntargets, long long total, int ts, int band,
                      double* band_pool, const double* scale, int* err, cudaStream_t st);
int launch_split_update(const void* tm_hi, const void* tm_lo, const void* tm_c, int ts, int nt,
                        int band, int k, float* c_pool,
                        const float* inv_scale, int* err, cudaStream_t st, int max_ctas = 0);

}  // namespace egs
