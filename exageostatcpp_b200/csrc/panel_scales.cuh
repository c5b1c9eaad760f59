// Per-row scales and the two splittings of a solved panel row used by the
// mixed-precision updates: FP16 hi/lo parts for the split-FP16 tcgen05 update
// and signed 7-bit slices for the Ozaki int8 products.  Shared by the slicing
// kernels (ozaki_band.cu) and the FP16 split of the DMMA form (split_gemm.cu).
#pragma once
#include <cuda_fp16.h>
#include <cstdint>

namespace egs {

constexpr int kOzSlices = 7;  // signed 7-bit slices per value (2^-49 of the row maximum)
// Slices of the off-band panel solve (FP32-stored rows times rows of L_kk^-1):
// 2^-42 of the row maxima.  The product with the inverse can cancel by the
// size of L_kk^-1's entries (10^4 to 10^5 for smooth kernels), which 2^-42
// still keeps below the FP32 rounding the solved rows get in storage.
constexpr int kOzPanelSlices = 6;

// FP16 split scale of a row with maximum m: inv_scale = 2^(e - 13) for
// 2^e <= m < 2^(e+1), so the scaled row lies below 2^14; rows whose maximum is
// 0 (or below 2^-120) get 0 and split to zeros; NaN or Inf rows get NaN.
__device__ __forceinline__ float f16_row_inv_scale(double m) {
  const long long bits = __double_as_longlong(m);
  const int e = (int)((bits >> 52) & 0x7FF) - 1023;
  if (e == 1024) return __int_as_float(0x7fc00000);  // NaN or Inf in the row: propagate
  if (!(m > 0.0) || e < -120) return 0.0f;
  return __int_as_float((e - 13 + 127) << 23);  // 2^(e-13), finite for e <= 140
}

// Ozaki row scale: 2^e with m < 2^e (the scaled row lies in (-1, 1)); 0 rows
// get 0, NaN rows NaN.
__device__ __forceinline__ double oz_row_scale(double m) {
  if (!(m > 0.0)) return (m == 0.0) ? 0.0 : __longlong_as_double(0x7ff8000000000000ll);
  const long long bits = __double_as_longlong(m);
  const int e = (int)((bits >> 52) & 0x7FF) - 1023;  // 2^e <= m < 2^(e+1) for normal m
  return (e >= 1023) ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(1.0, e + 1);
}

// The first NP (at most seven) signed 7-bit slices of 16 scaled values
// (|v| < 1), one 16-byte store per slice: slice p (1..NP) of v is sign(v) * (floor(|v| 2^(7p)) mod 2^7),
// read off the truncated 49-bit fixed-point magnitude floor(|v| 2^49), which
// is the double's significand shifted by its exponent.  These are the values
// the repeated exact steps a_p = trunc(2^7 v), v <- 2^7 v - a_p give; the
// integer form keeps the slicing off the FP64 pipe.  Zero, subnormal and
// non-finite inputs give zero slices.
//
// Four values at a time: 28 bits of a magnitude are spread to one slice per
// byte, a 4 x 4 byte transpose brings the values of a slice together, and the
// signs go on whole words: s in 0..127 becomes -s as (0x80 - s) ^ 0x80, without
// carries between bytes.  Byte by byte the mixed evaluation of N = 20,011 took 30.87 ms,
// so 30.60.
__device__ __forceinline__ unsigned oz_prmt(unsigned a, unsigned b, unsigned sel) {
  unsigned d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

__device__ __forceinline__ unsigned oz_spread7(unsigned x) {  // bits 7i .. 7i+6 to byte i
  return (x & 0x7Fu) | ((x << 1) & 0x7F00u) | ((x << 2) & 0x7F0000u) | ((x << 3) & 0x7F000000u);
}

template <int NP = kOzSlices>
__device__ __forceinline__ void oz_emit_slices(const double (&v)[16], int8_t* dst, long long slice_stride) {
  static_assert(NP >= 1 && NP <= kOzSlices, "slices of the 49-bit magnitude");
  unsigned out[NP][4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    unsigned lo[4], hi[4], top[4];  // slices 7..4 and 3..1 of each value, lowest byte first; sign words
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const unsigned long long b = (unsigned long long)__double_as_longlong(v[4 * g + c]);
      const int ex = (int)((b >> 52) & 0x7FF);
      const unsigned long long sig = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
      const int sh = 1026 - ex;  // |v| = sig 2^(ex - 1075), so floor(|v| 2^49) = sig >> (1026 - ex)
      const unsigned long long mag = (ex == 0 || ex > 1022 || sh > 52) ? 0ull : (sig >> sh);
      lo[c] = oz_spread7((unsigned)mag);
      hi[c] = oz_spread7((unsigned)(mag >> 28));
      top[c] = (unsigned)(b >> 32);
    }
    // 0xFF in the bytes of negative values (selectors 0xB and 0xF copy the sign of byte 3)
    const unsigned neg = oz_prmt(oz_prmt(top[0], top[1], 0xFBu), oz_prmt(top[2], top[3], 0xFBu), 0x5410u);
#pragma unroll
    for (int p = 1; p <= NP; ++p) {
      const unsigned* w = p >= 4 ? lo : hi;
      const int byte = p >= 4 ? 7 - p : 3 - p;
      const unsigned pair = byte < 2 ? 0x5140u : 0x7362u, half = (byte & 1) ? 0x7632u : 0x5410u;
      const unsigned s = oz_prmt(oz_prmt(w[0], w[1], pair), oz_prmt(w[2], w[3], pair), half);
      const unsigned m = (0x80808080u - s) ^ 0x80808080u;
      out[p - 1][g] = (m & neg) | (s & ~neg);
    }
  }
#pragma unroll
  for (int p = 0; p < NP; ++p)
    *reinterpret_cast<uint4*>(dst + p * slice_stride) = make_uint4(out[p][0], out[p][1], out[p][2], out[p][3]);
}

// hi = fp16(v), lo = fp16(v - hi) of 16 scaled values, two 16-byte stores each.
__device__ __forceinline__ void f16_emit_split(const double (&v)[16], __half* hi, __half* lo) {
  union {
    __half h[16];
    int4 q[2];
  } H, L;
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    const __half h = __double2half(v[c]);
    H.h[c] = h;
    L.h[c] = __double2half(v[c] - (double)__half2float(h));
  }
  reinterpret_cast<int4*>(hi)[0] = H.q[0];
  reinterpret_cast<int4*>(hi)[1] = H.q[1];
  reinterpret_cast<int4*>(lo)[0] = L.q[0];
  reinterpret_cast<int4*>(lo)[1] = L.q[1];
}

}  // namespace egs
