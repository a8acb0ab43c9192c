// FP64 tensor-core product step shared by the kernels that contract in double precision.
#pragma once

namespace sincgpu {

// D (8 x 8, two values per lane) += A (8 x 4) B (4 x 8) on the FP64 tensor cores;
// lane g * 4 + t holds A[g][t], B[t][g] and D[g][2t], D[g][2t + 1]
__device__ __forceinline__ void dmma_884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

}  // namespace sincgpu
