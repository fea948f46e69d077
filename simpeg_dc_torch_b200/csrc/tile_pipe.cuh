// 64 x NC products with a long K: the operands of K stages of kPipeK columns
// are copied (cp.async) kPipeSlots - 1 stages ahead into a ring in shared
// memory, one barrier per stage.  Double products run on the tensor cores
// (SmallTile, solve_small.cuh).
//
// Bound by the double rate (37 TFLOP/s): a stage of 64 x 64 x 16 is 1,024
// cycles of it against 16 KB of copies; 52 KB of ring let three CTAs share an
// SM and hide one another's barriers (a fourth slot, or two CTAs, were slower).
// Measured on a B200, the widest trailing update of the 269,001-node benchmark
// (14,160 tiles, K = 256): 26 TFLOP/s; the float64 trailing updates of a
// factorization 34.3 -> 20.5 ms, the substitution products of two solves 25.7 ->
// 13.6 ms against 64 x 64 register tiles loaded between barriers, one panel
// per update.
#pragma once
#include <cuda_runtime.h>

#include "solve_small.cuh"

namespace dct {
namespace {

constexpr int kPipeK = 16, kPipeSlots = 3;

template <typename T, int NC, bool MK>
struct TilePipe {
  // A as [k][m] (64 rows and padding) or [m][k]; B as [k][n]
  static constexpr int LA = MK ? kPipeK + 4 : kPanel + 4;
  static constexpr int EA = MK ? kPanel * LA : kPipeK * LA;
  static constexpr int EB = kPipeK * (NC + 4);
  static constexpr int kElems = kPipeSlots * (EA + EB);

  // acc += A B over K columns; a(dst, kw) and b(dst, kw) copy the next kw
  // columns of their operand, zeros to the next multiple of 4.  All of `ring`
  // is free again when it returns.
  template <typename SA, typename SB>
  static __device__ __forceinline__ void run(T* ring, int K, int rows, int cols,
                                             SmallTile<T, NC>& acc, SA& a, SB& b) {
    const int nst = (K + kPipeK - 1) / kPipeK;
    auto issue = [&](int st) {
      if (st < nst) {
        T* slot = ring + st % kPipeSlots * (EA + EB);
        const int kw = min(kPipeK, K - st * kPipeK);
        a(slot, kw);
        b(slot + EA, kw);
      }
      small_commit();
    };
    for (int st = 0; st < kPipeSlots - 1; ++st) issue(st);
    for (int st = 0; st < nst; ++st) {
      small_wait<kPipeSlots - 2>();
      __syncthreads();   // stage st has landed, stage st - 1 is read
      issue(st + kPipeSlots - 1);
      const T* slot = ring + st % kPipeSlots * (EA + EB);
      const int kw = K - st * kPipeK;
      if (kw >= kPipeK)
        acc.template mul<MK>(slot, LA, slot + EA, kPipeK, rows, cols);
      else
        acc.template mul<MK>(slot, LA, slot + EA, (kw + 3) & ~3, rows, cols);
    }
    small_wait<0>();
    __syncthreads();
  }
};

// Operand streams.  Every thread keeps the addresses of its copies of a stage
// and moves them on by a constant: computed anew for each stage, they took as
// many issue slots as the products (sm__inst_issued 47 % at 55 % of the double
// tensor rate; now 39 % at 68 %, 2,228 tiles of a 75,843-node case).  Rows and columns beyond the tile repeat its last one, which
// only reaches entries that nothing keeps; columns beyond K are zeros.

// [k][m]: 64 rows of the columns of a column-major matrix
template <typename T, int W>
struct ColStream {
  static_assert(W == kPanel, "two rows per lane");
  const T* p;
  int64_t ld;
  int up;   // from the first row of the thread to its second
  __device__ __forceinline__ ColStream(const T* src, int64_t ld_, int nr) : ld(ld_) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = min(lane, nr - 1);
    p = src + warp * ld + r;
    up = min(lane + 32, nr - 1) - r;
  }
  __device__ __forceinline__ void operator()(T* dst, int kw) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* d = dst + warp * (kPanel + 4) + lane;
#pragma unroll
    for (int c = 0; c < kPipeK; c += 8) {
      const bool in = warp + c < kw;
      const T* q = in ? p + c * ld : p;
      if (in || warp + c < ((kw + 3) & ~3)) {
        small_copy<sizeof(T)>(d + c * (kPanel + 4), q, in);
        small_copy<sizeof(T)>(d + c * (kPanel + 4) + 32, q + up, in);
      }
    }
    p += kPipeK * ld;
  }
};

// [m][k]: the rows of nm columns of a column-major matrix
template <typename T>
struct RowStream {
  const T* p[4];
  __device__ __forceinline__ RowStream(const T* src, int64_t ld, int nm) {
    static_assert(kPipeK == 16 && kThreads == 256, "half a warp per column");
#pragma unroll
    for (int i = 0; i < 4; ++i)
      p[i] = src + min((int(threadIdx.x) >> 4) + 16 * i, nm - 1) * ld + (threadIdx.x & 15);
  }
  __device__ __forceinline__ void operator()(T* dst, int kw) {
    const int k = threadIdx.x & 15;
    T* d = dst + (threadIdx.x >> 4) * (kPipeK + 4) + k;
    if (k < ((kw + 3) & ~3)) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        small_copy<sizeof(T)>(d + 16 * i * (kPipeK + 4), k < kw ? p[i] : p[i] - k, k < kw);
        p[i] += kPipeK;
      }
    }
  }
};

// rows of an (n, k) buffer, columns j0 .. j0 + rc - 1: row0, row0 + 1, ... or,
// with a list, rows[0], rows[1], ...  V: elements per copy.
template <typename T, int NC, int V, bool LIST>
struct RhsStream {
  static constexpr int U = NC / V, R = kThreads / U;   // copies a row, rows at a time
  const T* p;
  const int32_t* rows;
  int k, r;
  __device__ __forceinline__ RhsStream(const T* src, int k_, int j0, int rc, int64_t row0,
                                       const int32_t* rows_)
      : rows(rows_), k(k_) {
    r = threadIdx.x / U;
    p = src + j0 + min(int(threadIdx.x) % U * V, rc - V);
    if constexpr (!LIST) p += (row0 + r) * k;
  }
  __device__ __forceinline__ void operator()(T* dst, int kw) {
    T* d = dst + r * (NC + 4) + threadIdx.x % U * V;
#pragma unroll
    for (int c = 0; c < kPipeK; c += R) {
      const bool in = r + c < kw;
      if (in || r + c < ((kw + 3) & ~3)) {
        const T* q = p;
        if (in) q = LIST ? p + int64_t(rows[r + c]) * k : p + int64_t(c) * k;
        small_copy<V * sizeof(T)>(d + c * (NC + 4), q, in);
      }
    }
    if constexpr (LIST)
      rows += kPipeK;
    else
      p += int64_t(kPipeK) * k;
  }
};

// acc of one tile less that of another
template <typename Tile>
__device__ __forceinline__ void tile_subtract(Tile& x, const Tile& y) {
  using E = typename Tile::Elem;
  constexpr int n = sizeof(x.a) / sizeof(E);
  E* xp = reinterpret_cast<E*>(&x.a);
  const E* yp = reinterpret_cast<const E*>(&y.a);
#pragma unroll
  for (int i = 0; i < n; ++i) xp[i] -= yp[i];
}

}  // namespace
}  // namespace dct
