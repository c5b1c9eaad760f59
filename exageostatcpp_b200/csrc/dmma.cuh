// FP64 tensor-core (mma.sync m16n8k16 .f64) and global memory helpers of
// the DMMA kernels.  Fragment layout of one warp (g = lane / 4, t = lane % 4):
//   A: a[2j], a[2j+1] = rows g, g + 8 at k = t + 4j      (j = 0..3)
//   B: b[i]           = column g at k = t + 4i           (i = 0..3)
//   C: c[h], c[2+h]   = rows g, g + 8 at column 2t + h   (h = 0, 1)
#pragma once
#include <cstdint>

namespace egs {

__device__ __forceinline__ void ldg_v2f64(const double* p, double& a, double& b) {
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p));
}
__device__ __forceinline__ void stg_v2f64(double* p, double a, double b) {
  asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ void dmma_16816(double (&d)[4], const double (&a)[8], const double (&b)[4]) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
        "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// K = 8: A a[2j], a[2j+1] = rows g, g + 8 at k = t + 4j (j = 0, 1), B b[i] = column g at k = t + 4i.
__device__ __forceinline__ void dmma_1688(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

}  // namespace egs
