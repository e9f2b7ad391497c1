// The FP64 tensor-core products of the accumulation, product and FFT-branch kernels.
#pragma once
#include <cuda_runtime.h>

namespace spx {

// D(16x8) += A(16x8) B(8x8), f64. Fragments: a[2q+h] = A(g+8h, t+4q), b[q] = B(t+4q, g),
// d[r] = D(g + 8*(r>>1), 2t + (r&1)); g = lane/4, t = lane%4.
__device__ __forceinline__ void dmma_16x8x8(double (&d)[4], const double* a, const double* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// D(8x8) += A(8x4) B(4x8), f64: a = A(g, t), b = B(t, g), d[r] = D(g, 2t + r).
__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

}  // namespace spx
