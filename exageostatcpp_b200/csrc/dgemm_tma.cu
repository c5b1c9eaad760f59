// FP64 tensor-core update  C := C - A * B^T  on the tile-major lower storage,
// fed by TMA, for sm_100a.
//
// This is the trailing syrk/gemm of the tiled Cholesky (the N^3/3 part of
// CHAMELEON_dpotrf_Tile, ChameleonDense.cpp:25-37) and, with K = 64 or 128, the
// updates between the outer blocks of a panel.
//
// Geometry.  Every operand row is a *global* matrix row g in [0, Np); its data
// lives in tile row g / ts at local row g % ts.  A and B take their K columns
// from one tile column (a_tcol / b_tcol) starting at a local column offset; C is
// addressed element by element through (global row, global column) and
// elements of upper tiles are never written.  Because ts is a multiple of 64,
// a 16-row TMA box never straddles two tiles, so a CTA tile may span tile
// boundaries.
//
// Work unit.  One CTA computes one C tile (64 x 64, smaller where that would leave
// SMs idle, gemm_tile_shape) and exits; four CTAs share an SM, so one tile's C
// round trip and pipeline fill run beside the other tiles' MMAs, and the
// hardware balances the triangular tile set.  FP64-tensor bound: 33.5 TF/s on the
// N = 40,000 trailing updates (K = 960; cuBLAS DGEMM about 35.4) and 27.3 at
// N = 10,000; one persistent 128 x 128 CTA per SM (its epilogue uncovered, whole
// tiles as the unit of the last wave) reached 27.9 and 20.3, 128 x 64 tiles at two
// CTAs per SM 31.6 and 25.2.
//
// Pipeline.  Warp 0 issues 3-D TMA loads (16 rows x 16 columns x tile-slot, one box
// per lane) two stages ahead into a ring of 16-column 128B-swizzled shared-memory
// stages guarded by mbarriers; the four warps, one per SM sub-partition, run
// mma.sync m16n8k16 .f64 (the FP64 tensor path of sm_100a: one warp keeps its
// sub-partition's pipe full, 128 cycles per instruction).  The 16 rows of an MMA
// fragment are mapped to tile rows through fixed permutations chosen so that
// every fragment load is free of shared-memory bank conflicts under the 128-byte
// swizzle (A: 16-byte loads of row pairs; B: 8-byte loads).
//
// Every wait is bounded: a thread that polls longer than the limit records an
// error in *err and leaves; the host turns that into EGS_ERR_TIMEOUT.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cstdint>
#include "common.cuh"
#include "dmma.cuh"
#include "kernels.cuh"
#include "mbarrier.cuh"

namespace egs {

namespace gemm {
constexpr int BK = 16;                                // columns per stage = one MMA k-step
constexpr int WARPS = 4;                              // 2 x 2 warp tiles; warp 0 also issues the TMA loads
constexpr int THREADS = WARPS * 32;
constexpr int LEAD = 2;                               // stages issued ahead of the one being consumed
constexpr int BOX_ROWS = 16;                          // 16 doubles = one 128-byte swizzle row
constexpr int BOX_BYTES = BOX_ROWS * BK * 8;          // 16 rows x BK columns
constexpr int GROUP_COLS = 1024;                      // columns per raster group

// Tile shape (GemmDesc::cfg): 0 = 64 x 64, 1 = 64 x 32, 2 = 32 x 32.
__host__ __device__ constexpr int block_m(int cfg) { return cfg == 2 ? 32 : 64; }
__host__ __device__ constexpr int block_n(int cfg) { return cfg == 0 ? 64 : 32; }
template <int CFG>
struct Shape {
  static constexpr int BM = block_m(CFG), BN = block_n(CFG);
  static constexpr int STAGES = CFG == 0 ? 3 : 4;
  static constexpr int CTAS = 4;                      // per SM, at most 128 registers per thread
  static constexpr int MI = BM / 32, NI = BN / 16;    // 16 x 8 MMA tiles per warp
  static constexpr int BOXES = (BM + BN) / BOX_ROWS;
  static constexpr int STAGE_BYTES = BOXES * BOX_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 2 * STAGES * 8 + 1024;
};
}  // namespace gemm

// MMA row g (0..7) of an A fragment -> tile row 2*perm[g] within a 16-row box;
// row g+8 -> the next row, so (a_2j, a_2j+1) is one 16-byte load.
__device__ __forceinline__ int perm_a(int g) { return ((g & 1) << 2) | (g >> 1); }
// MMA row r (0..15) of a B fragment (the n index) -> tile row within a 16-row box.
__device__ __forceinline__ int perm_b(int r) {
  return (r & 1) | (((r >> 2) & 1) << 1) | (((r >> 1) & 1) << 3) | (((r >> 3) & 1) << 2);
}

// Raster: groups of GROUP_COLS columns; inside a group, block-rows outer,
// block-columns inner, so a group's B panel stays in L2 while A streams once.
// A lower problem's group starts at the first block-row that reaches its columns.
__host__ __device__ inline int group_first_row(const GemmDesc& d, int nb0) {
  return d.lower ? nb0 * gemm::block_n(d.cfg) / gemm::block_m(d.cfg) : 0;
}

__device__ __forceinline__ void decode_block(long long L, const GemmDesc& d, int& mb, int& nb) {
  const int group = gemm::GROUP_COLS / gemm::block_n(d.cfg);
  mb = d.MB;
  nb = d.NB;
  for (int nb0 = 0; nb0 < d.NB; nb0 += group) {
    const int ge = min(group, d.NB - nb0);
    const int mstart = group_first_row(d, nb0);
    const long long cnt = (long long)ge * (d.MB - mstart);
    if (L < cnt) {
      mb = mstart + (int)(L / ge);
      nb = nb0 + (int)(L % ge);
      return;
    }
    L -= cnt;
  }
}

// Blocks with nothing to write: above the diagonal, or (band targets of the
// lower pool, c_mode 2) wholly below the band.
__device__ __forceinline__ bool block_skipped(const GemmDesc& d, int mb, int nb) {
  const int bm = gemm::block_m(d.cfg), bn = gemm::block_n(d.cfg);
  if (mb >= d.MB || nb >= d.NB) return true;
  if (d.lower && (mb + 1) * bm <= nb * bn) return true;
  if (d.c_mode != 2) return false;
  const int ti = (d.c_row0 + mb * bm) / d.ts, tj = (d.c_col0 + nb * bn + bn - 1) / d.ts;
  return ti - tj > d.c_band;
}

// C(gi, gj) sits at row part + column part: tiles of one column are contiguous.
__device__ __forceinline__ long long c_row_part(const GemmDesc& d, int gi, int& ti) {
  ti = gi / d.ts;
  return (long long)ti * d.ts * d.ts + (gi - ti * d.ts);
}
__device__ __forceinline__ long long c_col_part(const GemmDesc& d, int gj, int& tj) {
  tj = gj / d.ts;
  const long long slot0 = d.c_mode != 1 ? d.tile_base + tile_slot(tj, tj, d.nt) - tj
                                        : (long long)(d.c_tile_off + tj) * (d.c_band + 1) - tj;
  return slot0 * d.ts * d.ts + (long long)(gj - tj * d.ts) * d.ts;
}
__device__ __forceinline__ bool c_written(const GemmDesc& d, int ti, int tj) {
  return ti >= tj && (d.c_mode == 0 || ti - tj <= d.c_band);
}

template <int CFG, bool kBatched>
__global__ void __launch_bounds__(gemm::THREADS, gemm::Shape<CFG>::CTAS)
dgemm_update_kernel(const __grid_constant__ CUtensorMap tmap, double* __restrict__ tiles,
                    const __grid_constant__ GemmDesc single, GemmJobs J, int* __restrict__ err) {
  using namespace gemm;
  using S = Shape<CFG>;
  constexpr int BM = S::BM, BN = S::BN, STAGES = S::STAGES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // the job of this block, and its tile (job tables are constant)
  const GemmDesc* dp = &single;
  long long L = blockIdx.x;
  if constexpr (kBatched) {
    int lo = 0, hi = J.njobs - 1;
    while (lo < hi) {  // last job with begin <= L
      const int mid = (lo + hi + 1) >> 1;
      if (J.begin[mid] <= L) lo = mid; else hi = mid - 1;
    }
    L -= J.begin[lo];
    dp = J.jobs + lo;
  }
  const GemmDesc& d = *dp;
  int mb, nb;
  decode_block(L, d, mb, nb);
  if (block_skipped(d, mb, nb)) {
    grid_dependency_wait();
    return;
  }
  // 1024-byte aligned stage base (128B-swizzle atoms), kept as an offset into the
  // shared array so every access stays a shared-memory access.
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * S::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  grid_dependency_wait();
  const int ksteps = d.K / BK;

  // Producer state: lane b of warp 0 loads box b of every stage (A boxes first).
  int x = d.ts, z = 0, y0 = 0;  // fully out of bounds -> zero fill
  if (warp == 0 && lane < S::BOXES) {
    const bool is_a = lane < BM / BOX_ROWS;
    const int g0 = is_a ? d.a_row0 + mb * BM + lane * BOX_ROWS : d.b_row0 + nb * BN + (lane - BM / BOX_ROWS) * BOX_ROWS;
    y0 = is_a ? d.a_col0 : d.b_col0;
    if (g0 < d.np) {
      const int tg = g0 / d.ts;
      x = g0 - tg * d.ts;
      z = (int)(d.tile_base + tile_slot(tg, is_a ? d.a_tcol : d.b_tcol, d.nt));
    }
  }
  // Issues stage j (warp 0, all lanes); its slot was last used by stage j - STAGES.
  auto issue = [&](int j) {
    const int sj = j % STAGES;
    bool slot_free = true;
    if (lane == 0) {
      slot_free = mbar_wait(&empty[sj], ((j / STAGES) & 1) ^ 1, err);
      if (slot_free) mbar_expect_tx(&full[sj], S::STAGE_BYTES);
    }
    if (!__shfl_sync(0xffffffffu, (int)slot_free, 0)) return false;
    if (lane < S::BOXES)
      tma_load_3d(smem + sj * S::STAGE_BYTES + lane * BOX_BYTES, &tmap, &full[sj], x, y0 + j * BK, z);
    return true;
  };
  int issued = 0;  // stages whose copies are under way (warp 0)
  if (warp == 0)
    while (issued < min(LEAD, ksteps) && issue(issued)) ++issued;

  const int g = lane >> 2, t = lane & 3;
  const int wm = warp & 1, wn = warp >> 1;  // warp sub-tile: rows wm*BM/2.., cols wn*BN/2..
  const int pa = perm_a(g);
  // Byte offsets (inside one 16-row box) of this thread's fragment elements.
  int aoff[4], boff[2][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int k = t + 4 * j;
    aoff[j] = k * 128 + ((pa ^ (k & 7)) << 4);
  }
#pragma unroll
  for (int sN = 0; sN < 2; ++sN) {
    const int fb = perm_b(g + 8 * sN);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = t + 4 * i;
      boff[sN][i] = k * 128 + (((fb >> 1) ^ (k & 7)) << 4) + ((fb & 1) << 3);
    }
  }
  {
    // this warp's part of C to L2: one column per lane, 16 rows (128 bytes) per request
    const int nl = nb * BN + wn * (BN / 2) + (lane & (BN / 2 - 1));
    int tj;
    const long long cp = c_col_part(d, d.c_col0 + nl, tj);
#pragma unroll
    for (int mi = 0; mi < S::MI; ++mi) {
      const int ml = mb * BM + wm * (BM / 2) + mi * 16;
      int ti;
      const long long p = c_row_part(d, d.c_row0 + ml, ti) + cp;
      if (nl < d.N && ml < d.M && c_written(d, ti, tj)) asm volatile("prefetch.global.L2 [%0];" ::"l"(tiles + p));
    }
  }
  double acc[S::MI][S::NI][4];
#pragma unroll
  for (int mi = 0; mi < S::MI; ++mi)
#pragma unroll
    for (int ni = 0; ni < S::NI; ++ni)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[mi][ni][q] = 0.0;

  bool ok = true;
  int s = 0, ph = 0;
#pragma unroll 1
  for (int kt = 0; kt < ksteps; ++kt) {
    if (warp == 0 && kt + LEAD < ksteps && issued == kt + LEAD && issue(issued)) ++issued;
    if (!mbar_wait(&full[s], ph, err)) {
      ok = false;
      break;
    }
    const uint8_t* sa = smem + s * S::STAGE_BYTES + wm * (BM / 2 / BOX_ROWS) * BOX_BYTES;
    const uint8_t* sb = smem + s * S::STAGE_BYTES + (BM / BOX_ROWS + wn * (BN / 2 / BOX_ROWS)) * BOX_BYTES;
    double bf[S::NI][4];
#pragma unroll
    for (int ni = 0; ni < S::NI; ++ni)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        bf[ni][i] = *reinterpret_cast<const double*>(sb + (ni >> 1) * BOX_BYTES + boff[ni & 1][i]);
#pragma unroll
    for (int mi = 0; mi < S::MI; ++mi) {
      double af[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 v = *reinterpret_cast<const double2*>(sa + mi * BOX_BYTES + aoff[j]);
        af[2 * j] = v.x;
        af[2 * j + 1] = v.y;
      }
#pragma unroll
      for (int ni = 0; ni < S::NI; ++ni) dmma_16816(acc[mi][ni], af, bf[ni]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (++s == STAGES) {
      s = 0;
      ph ^= 1;
    }
  }
  if (!ok) {
    // Drain: every stage this CTA issued must have landed before it exits.
    if (threadIdx.x == 0)
      for (int j = (issued > STAGES ? issued - STAGES : 0); j < issued; ++j)
        mbar_wait(&full[j % STAGES], (j / STAGES) & 1, err);
    return;
  }

  grid_dependents_launch();
  // Epilogue: C -= acc; element pairs (row, row+1) are contiguous in a column.
  // Per n8 block all loads are issued before any store.
  long long rp[S::MI];
  int ti[S::MI];
#pragma unroll
  for (int mi = 0; mi < S::MI; ++mi) {
    const int ml = mb * BM + wm * (BM / 2) + mi * 16 + 2 * pa;
    rp[mi] = c_row_part(d, d.c_row0 + ml, ti[mi]);
    if (ml >= d.M) ti[mi] = -1;  // above every tile column: not written
  }
#pragma unroll
  for (int ni = 0; ni < S::NI; ++ni) {
    double* ptr[2][S::MI];
    double cv[2][S::MI][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int nl = nb * BN + wn * (BN / 2) + (ni >> 1) * 16 + perm_b(2 * t + 8 * (ni & 1)) + h;
      int tj;
      const long long cp = c_col_part(d, d.c_col0 + nl, tj);
#pragma unroll
      for (int mi = 0; mi < S::MI; ++mi) {
        ptr[h][mi] = (nl < d.N && c_written(d, ti[mi], tj)) ? tiles + (rp[mi] + cp) : nullptr;
        if (ptr[h][mi]) ldg_v2f64(ptr[h][mi], cv[h][mi][0], cv[h][mi][1]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int mi = 0; mi < S::MI; ++mi)
        if (ptr[h][mi])
          stg_v2f64(ptr[h][mi], cv[h][mi][0] - acc[mi][ni][h], cv[h][mi][1] - acc[mi][ni][2 + h]);
  }
}

// One-time lookups below use function-local statics, whose initialisation is
// thread-safe: problems may be created from several host threads at once.
int tensor_map_encoder(void** fn_out) {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    cudaDriverEntryPointQueryResult q;
    void* f = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !f) {
      cudaGetLastError();
      return nullptr;
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }();
  if (!fn) {
    set_last_error("cuTensorMapEncodeTiled unavailable", "tensor_map_encoder");
    return EGS_ERR_CUDA;
  }
  *fn_out = reinterpret_cast<void*>(fn);
  return EGS_OK;
}

int gemm_init_tensor_map(void* tmap_storage, double* tiles, int ts, long long ntiles) {
  void* fn = nullptr;
  if (tensor_map_encoder(&fn) != EGS_OK) return EGS_ERR_CUDA;
  if (ts % 64 != 0 || ((uintptr_t)tiles & 15) != 0) return EGS_ERR_INVALID;
  cuuint64_t dims[3] = {(cuuint64_t)ts, (cuuint64_t)ts, (cuuint64_t)ntiles};
  cuuint64_t strides[2] = {(cuuint64_t)ts * 8, (cuuint64_t)ts * ts * 8};
  cuuint32_t box[3] = {gemm::BOX_ROWS, gemm::BK, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  auto encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  CUresult r = encode(reinterpret_cast<CUtensorMap*>(tmap_storage), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, tiles,
                        dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled failed", "gemm_init_tensor_map");
    return EGS_ERR_CUDA;
  }
  return EGS_OK;
}

int gemm_num_sms() {
  static const int sms = []() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
  }();
  return sms;
}

static void set_gemm_smem_attributes() {
  static std::once_flag done[64];
  once_per_device(done, []() {
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(dgemm_update_kernel<0, false>, attr, gemm::Shape<0>::SMEM_BYTES);
    cudaFuncSetAttribute(dgemm_update_kernel<0, true>, attr, gemm::Shape<0>::SMEM_BYTES);
    cudaFuncSetAttribute(dgemm_update_kernel<1, false>, attr, gemm::Shape<1>::SMEM_BYTES);
    cudaFuncSetAttribute(dgemm_update_kernel<1, true>, attr, gemm::Shape<1>::SMEM_BYTES);
    cudaFuncSetAttribute(dgemm_update_kernel<2, false>, attr, gemm::Shape<2>::SMEM_BYTES);
    cudaFuncSetAttribute(dgemm_update_kernel<2, true>, attr, gemm::Shape<2>::SMEM_BYTES);
  });
}

// Tile shape of a launch of `total` 64 x 64 tiles.  The large tile reads least from
// L2 and wins once every SM has four of them (N = 40,000 trailing updates: 33.5
// TF/s against 32.3 with 64 x 32 and 30.8 with 32 x 32); a smaller launch is
// bound by the K loop of its one or two tiles per SM, which a smaller tile
// shortens (band approximation N = 10,000, tile 320, about 340 tiles a launch: 1.16 ms
// of updates with 64 x 32, 1.47 / 1.29 with the others; N = 1,600, 15 to 210
// tiles: 104 us with 32 x 32, 115 / 147 with the larger ones).
int gemm_tile_shape(long long total) {
  const long long sms = gemm_num_sms();
  return total < sms ? 2 : total < 4 * sms ? 1 : 0;
}

void finish_desc(GemmDesc& d) {
  using namespace gemm;
  d.MB = (d.M + block_m(d.cfg) - 1) / block_m(d.cfg);
  d.NB = (d.N + block_n(d.cfg) - 1) / block_n(d.cfg);
  const int group = GROUP_COLS / block_n(d.cfg);
  long long total = 0;
  for (int nb0 = 0; nb0 < d.NB; nb0 += group) {
    const int ge = (d.NB - nb0) < group ? (d.NB - nb0) : group;
    total += (long long)ge * (d.MB - group_first_row(d, nb0));
  }
  d.total = total;
}

template <bool kBatched>
static int launch_cfg(int cfg, const void* tmap, double* tiles, const GemmDesc& d, const GemmJobs& J, long long total,
                      int* err, cudaStream_t st) {
  using namespace gemm;
  set_gemm_smem_attributes();
  const CUtensorMap& tm = *reinterpret_cast<const CUtensorMap*>(tmap);
  const char* where = "dgemm_update_kernel";
  const dim3 grid((unsigned)total), block(THREADS);
  if (cfg == 0) {
    dgemm_update_kernel<0, kBatched><<<grid, block, Shape<0>::SMEM_BYTES, st>>>(tm, tiles, d, J, err);
    return launch_status(where);
  }
  // Small launches overlap their set-up with the tail of the panel step before
  // them (N = 1,600: 605 -> 582 us per evaluation); large ones, and the panel steps
  // themselves, only take room from the tail they wait for (N = 10,000: 15.9 -> 16.1 ms).
  if (cfg == 1)
    return launch_overlapped(where, dgemm_update_kernel<1, kBatched>, grid, block, Shape<1>::SMEM_BYTES, st, tm, tiles,
                             d, J, err);
  return launch_overlapped(where, dgemm_update_kernel<2, kBatched>, grid, block, Shape<2>::SMEM_BYTES, st, tm, tiles, d,
                           J, err);
}

static int launch_desc(const void* tmap, double* tiles, GemmDesc& d, int* err, cudaStream_t st) {
  if (d.M <= 0 || d.N <= 0 || d.K <= 0) return EGS_OK;
  if (d.K % gemm::BK != 0) return EGS_ERR_INVALID;
  d.cfg = 0;
  finish_desc(d);
  if ((d.cfg = gemm_tile_shape(d.total)) != 0) finish_desc(d);
  return launch_cfg<false>(d.cfg, tmap, tiles, d, GemmJobs{nullptr, nullptr, 0, 0}, d.total, err, st);
}

// Trailing update of step k: C(i, j) -= L(i, k) L(j, k)^T for all k < j <= i, on the
// first `rows` rows and columns.
int launch_gemm_trailing(const void* tmap, double* tiles, int ts, int nt, int rows, int k, int* err, cudaStream_t st) {
  GemmDesc d{};
  d.ts = ts;
  d.nt = nt;
  d.np = nt * ts;
  const int r0 = (k + 1) * ts;
  d.M = d.N = rows - r0;
  d.K = ts;
  d.a_row0 = d.b_row0 = d.c_row0 = d.c_col0 = r0;
  d.a_col0 = d.b_col0 = 0;
  d.a_tcol = d.b_tcol = k;
  d.lower = 1;
  return launch_desc(tmap, tiles, d, err, st);
}

// Update of step k of the band approximation: tiles (m, c), k < c < k + band,
// c <= m < c + band, in one launch, on the first `rows` rows and columns.
int launch_gemm_band(const void* tmap, double* tiles, int ts, int nt, int rows, int k, int band, int* err,
                     cudaStream_t st) {
  GemmDesc d{};
  d.ts = ts;
  d.nt = nt;
  d.np = nt * ts;
  const int r0 = (k + 1) * ts;
  const int cend = nt < k + band ? nt : k + band;               // columns: tiles k+1 .. cend-1
  const int rend = nt < cend - 1 + band ? nt : cend - 1 + band;  // rows: up to tile rend-1
  d.M = (rend * ts < rows ? rend * ts : rows) - r0;
  d.N = (cend * ts < rows ? cend * ts : rows) - r0;
  d.K = ts;
  d.a_row0 = d.b_row0 = d.c_row0 = d.c_col0 = r0;
  d.a_tcol = d.b_tcol = k;
  d.lower = 1;
  d.c_mode = 2;
  d.c_band = band - 1;
  return launch_desc(tmap, tiles, d, err, st);
}

// General form used by the panel factorisation (see kernels.cuh).
int launch_gemm_rows(const void* tmap, double* tiles, int ts, int nt, int M, int N, int K, int a_row0,
                     int a_col0, int a_tcol, int b_row0, int b_col0, int b_tcol, int c_row0, int c_col0,
                     int lower, int* err, cudaStream_t st) {
  GemmDesc d{};
  d.ts = ts;
  d.nt = nt;
  d.np = nt * ts;
  d.M = M;
  d.N = N;
  d.K = K;
  d.a_row0 = a_row0;
  d.a_col0 = a_col0;
  d.a_tcol = a_tcol;
  d.b_row0 = b_row0;
  d.b_col0 = b_col0;
  d.b_tcol = b_tcol;
  d.c_row0 = c_row0;
  d.c_col0 = c_col0;
  d.lower = lower;
  return launch_desc(tmap, tiles, d, err, st);
}

}  // namespace egs

namespace egs {

// One launch over many jobs (one per problem of a batch) of one tile shape cfg;
// jobs and begin live in device memory, begin[j] = number of blocks of jobs 0..j-1 (finish_desc totals).
int launch_gemm_batched(const void* tmap, double* tiles, int cfg, const GemmDesc* jobs, const long long* begin,
                        int njobs, long long total, int* err, cudaStream_t st) {
  if (njobs <= 0 || total <= 0) return EGS_OK;
  GemmDesc none{};
  return launch_cfg<true>(cfg, tmap, tiles, none, GemmJobs{jobs, begin, njobs, total}, total, err, st);
}

}  // namespace egs
