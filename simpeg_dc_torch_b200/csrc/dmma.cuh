// Double-precision tensor-core products (mma.sync m8n8k4): on B200 they run
// at the same 37 TFLOP/s as the FMA units (measured: 37.1 both, 128 threads
// per SM are enough), but one instruction takes the place of eight FMAs and
// an operand value loaded from shared memory serves eight products, so the
// shared-memory loads that bound a register-tiled product no longer do.
// Accumulation is in float64 with one rounding per product, as with fma().
//
// Fragments of a warp, g = lane / 4, t = lane % 4: A[g][t], B[t][g],
// C[g][2 t], C[g][2 t + 1].  An operand tile in shared memory, either
// [k][m] or [m][k], is read without bank conflicts when its leading
// dimension is 4 modulo 8.
#pragma once
#include <cuda_runtime.h>

namespace dct {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

}  // namespace dct
