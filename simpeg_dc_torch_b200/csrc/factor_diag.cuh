// The pivot test and its record, shared by the factor kernels.
#pragma once
#include <cuda_runtime.h>

#include "dct_internal.h"

namespace dct {
namespace {

__device__ __forceinline__ void flag_pivot(int* status, int s, int b) {
  if (atomicCAS(&status[0], 0, DCT_ERR_ZERO_PIVOT) == 0) {
    status[1] = s;
    status[2] = b;
  }
}

template <typename T>
__device__ __forceinline__ bool good_pivot(T v) {
  return v > T(0) && v < T(INFINITY);
}

}  // namespace
}  // namespace dct
