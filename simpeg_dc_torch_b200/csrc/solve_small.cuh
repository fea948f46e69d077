// Substitution with the supernodes of one panel (ns <= 64): one CTA per
// (supernode, system, NC right-hand sides).
//
//   forward   y = D^{-1} b (to B), then b[boundary rows] -= L_B y (atomics, A)
//   backward  x = D^{-T} (y - L_B^T x_B) (to A)
//
// D^{-1} and L_B are copied to shared memory column by column as they lie in
// HBM; the forward products read that image as [k][m], the backward ones as
// [m][k].  The double products run on the tensor cores (dmma.cuh).  What bounds
// the kernels is the latency of these copies and, in double, the products of
// the wide launches, so
//   - the shared memory of a launch is sized for its largest supernode (a
//     2-D leaf has 40 of the 64 columns), which lets more CTAs share an SM;
//   - NC follows the number of right-hand sides (8, 16, 32 or 64): 18 sources
//     in a 64-column tile are three quarters padding;
//   - the next launch of a pass starts early (programmatic dependent launch)
//     and copies its factors, which no launch of the pass writes, before it
//     waits for the predecessor's right-hand sides;
//   - a forward CTA whose right-hand sides are all zero writes y = 0 and is
//     done.  The sources and the adjoint sources of a survey are a few
//     electrodes, so most supernodes of the lower levels have none below them
//     (the test costs a dense right-hand side nothing: the tile has to arrive
//     before the product anyway).
// Measured on a B200, 56,525-node line, 12 systems, 186 sources, the two solves
// of an evaluation and gradient: 4.88 ms in double against 11.08 with 64-column
// register tiles loaded through registers and no test for zeros.
#pragma once
#include <cuda_runtime.h>

#include "dct_internal.h"
#include "dmma.cuh"

namespace dct {
namespace {

// a finished refinement: the remaining correction launches do nothing
__device__ __forceinline__ bool ir_skip(const int* skip) {
  return skip != nullptr && *reinterpret_cast<const volatile int*>(skip) != 0;
}

template <typename T>
__device__ __forceinline__ bool is_zero(const T& v) {
  return v == T(0);
}
template <>
__device__ __forceinline__ bool is_zero(const cplx& v) {
  return v.re == 0.0 && v.im == 0.0;
}

// 64 x NC output tile of a CTA of 256 threads.  mul adds A B over K columns
// (a multiple of 4), A read as [k][m] or (MK) [m][k], leading dimension la,
// B as [k][n], leading dimension NC + 4; only the first `rows` rows and
// `cols` columns of the tile need be right.  each(rows, f) visits this
// thread's entries f(row, column, value) of the first `rows` rows, rounded up.
template <typename T, int NC>
struct SmallTile {
  using Elem = T;
  static constexpr int JG = NC >= 16 ? 16 : 8, AG = kThreads / JG, P = 64 / AG, Q = NC / JG;
  T a[P][Q];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int q = 0; q < Q; ++q) a[p][q] = T(0);
  }
  template <bool MK, int NP>
  __device__ __forceinline__ void mul_np(const T* __restrict__ A, int la,
                                         const T* __restrict__ B, int K) {
    const int jg = threadIdx.x % JG, ag = threadIdx.x / JG;
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      T x[NP], y[Q];
#pragma unroll
      for (int p = 0; p < NP; ++p)
        x[p] = MK ? A[(ag + AG * p) * la + k] : A[k * la + ag + AG * p];
#pragma unroll
      for (int q = 0; q < Q; ++q) y[q] = B[k * (NC + 4) + jg + JG * q];
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int q = 0; q < Q; ++q) a[p][q] += x[p] * y[q];
    }
  }
  template <bool MK>
  __device__ __forceinline__ void mul(const T* A, int la, const T* B, int K, int rows, int) {
    const int np = (rows + AG - 1) / AG;
    if (np >= P) return mul_np<MK, P>(A, la, B, K);
    if constexpr (P > 1)
      if (np == 1) return mul_np<MK, 1>(A, la, B, K);
    if constexpr (P > 2) {
      if (np == 2) return mul_np<MK, 2>(A, la, B, K);
      mul_np<MK, 3>(A, la, B, K);
    }
  }
  template <typename Fn>
  __device__ __forceinline__ void each(int rows, Fn&& f) {
    const int jg = threadIdx.x % JG, ag = threadIdx.x / JG;
#pragma unroll
    for (int p = 0; p < P; ++p)
      if (AG * p < rows)
#pragma unroll
        for (int q = 0; q < Q; ++q) f(ag + AG * p, jg + JG * q, a[p][q]);
  }
};

// double: 8 x 8 tensor-core fragments; the row fragments are dealt out to the
// warps in turn, so that a supernode of few rows still occupies all of them
template <int NC>
struct SmallTile<double, NC> {
  using Elem = double;
  static constexpr int WM = NC == 64 ? 2 : (NC == 32 ? 4 : 8), WN = 8 / WM;
  static constexpr int MF = 8 / WM, NF = NC / 8 / WN, AG = 8;
  double a[MF][NF][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < MF; ++p)
#pragma unroll
      for (int q = 0; q < NF; ++q) a[p][q][0] = a[p][q][1] = 0.0;
  }
  template <bool MK, int NP>
  __device__ __forceinline__ void mul_np(const double* __restrict__ A, int la,
                                         const double* __restrict__ B, int K) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int m0 = 8 * (warp % WM) + g, n0 = 8 * NF * (warp / WM) + g;
    const double* pa = MK ? A + m0 * la + t : A + t * la + m0;
    const double* pb = B + t * (NC + 4) + n0;
    const int sa = MK ? 4 : 4 * la, sm = MK ? 8 * WM * la : 8 * WM;
#pragma unroll 4
    for (int k = 0; k < K; k += 4, pa += sa, pb += 4 * (NC + 4)) {
      double x[NP], y[NF];
#pragma unroll
      for (int p = 0; p < NP; ++p) x[p] = pa[p * sm];
#pragma unroll
      for (int q = 0; q < NF; ++q) y[q] = pb[8 * q];
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int q = 0; q < NF; ++q) dmma(a[p][q], x[p], y[q]);
    }
  }
  template <bool MK>
  __device__ __forceinline__ void mul(const double* A, int la, const double* B, int K, int rows,
                                      int cols) {
    const int warp = threadIdx.x >> 5, nfr = (rows + 7) / 8 - warp % WM;
    const int np = (nfr + WM - 1) / WM;
    if (nfr <= 0 || 8 * NF * (warp / WM) >= cols) return;
    if (np >= MF) return mul_np<MK, MF>(A, la, B, K);
    if constexpr (MF > 1)
      if (np == 1) return mul_np<MK, 1>(A, la, B, K);
    if constexpr (MF > 2) {
      if (np == 2) return mul_np<MK, 2>(A, la, B, K);
      mul_np<MK, 3>(A, la, B, K);
    }
  }
  template <typename Fn>
  __device__ __forceinline__ void each(int rows, Fn&& f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int p = 0; p < MF; ++p) {
      const int r = 8 * (warp % WM + WM * p);
      if (r < rows)
#pragma unroll
        for (int q = 0; q < NF; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            f(r + g, 8 * (NF * (warp / WM) + q) + 2 * t + h, a[p][q][h]);
    }
  }
};

// shared-memory places (in elements) of a launch whose supernodes have at
// most w columns and nb boundary rows
constexpr int kSmallRows = 1024;   // row indices kept at a time
template <typename T, int NC>
struct SmallPlaces {
  int ldd, ldl, lt, bt, rows;
  __host__ __device__ SmallPlaces(int w, int nb) {
    const int r = nb < kPanel ? nb : kPanel, most = w > r ? w : r;
    // the [m][k] products read whole row groups of the tile's threads
    constexpr int G = SmallTile<T, NC>::AG;
    const int wr = (w + G - 1) / G * G;
    ldd = ((w + 7) & ~7) + 4;      // 4 modulo 8, and room for the row padding
    ldl = ((r + 7) & ~7) + 4;
    lt = wr * ldd;                 // a tile of L_B, after D^{-1}
    bt = lt + wr * ldl;            // right-hand sides
    rows = bt + ((most + 3) & ~3) * (NC + 4);
  }
  __host__ __device__ size_t bytes(int nb) const {
    return sizeof(T) * size_t(rows) + 4 * size_t(nb < kSmallRows ? nb : kSmallRows);
  }
};

// one element (4, 8 or 16 bytes), or 16 bytes; zeros where it is not valid
template <int BYTES>
__device__ __forceinline__ void small_copy(void* dst, const void* src, bool valid) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  const int n = valid ? BYTES : 0;
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(d), "l"(src), "r"(n),
                 "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void small_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void small_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// nr x nc entries at src (column-major, ld sld) to dst[c * ld + r], zeros to
// the next multiples of 4
template <typename T>
__device__ __forceinline__ void small_load_cols(T* dst, int ld, const T* src, int64_t sld, int nr,
                                                int nc) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nr4 = (nr + 3) & ~3, nc4 = (nc + 3) & ~3;
  for (int c = warp; c < nc4; c += kThreads / 32)
    for (int r = lane; r < nr4; r += 32) {
      const bool in = r < nr && c < nc;
      small_copy<sizeof(T)>(dst + c * ld + r, in ? src + c * sld + r : src, in);
    }
}

// rows row(0) .. row(nr - 1), columns j0 .. j0 + rc - 1 of an (n, k) buffer to
// dst[r][j] (ld NC + 4), zeros to the next multiple of 4 rows and to column NC.
// wide: 16 bytes at a time (rows, j0 and rc allow it)
template <typename T, int NC, typename Row>
__device__ __forceinline__ void small_load_rhs(T* dst, const T* src, int k, int j0, int rc, int nr,
                                               bool wide, Row&& row) {
  const int nr4 = (nr + 3) & ~3;
  constexpr int V = 16 / sizeof(T);
  if (wide) {
    for (int q = threadIdx.x; q < nr4 * (NC / V); q += kThreads) {
      const int r = q / (NC / V), j = q % (NC / V) * V;
      const bool in = r < nr && j < rc;
      small_copy<16>(dst + r * (NC + 4) + j, in ? src + int64_t(row(r)) * k + j0 + j : src, in);
    }
  } else {
    for (int q = threadIdx.x; q < nr4 * NC; q += kThreads) {
      const int r = q / NC, j = q % NC;
      const bool in = r < nr && j < rc;
      small_copy<sizeof(T)>(dst + r * (NC + 4) + j, in ? src + int64_t(row(r)) * k + j0 + j : src,
                            in);
    }
  }
}

// CTAs per SM the kernels are compiled for: what a CTA waits for are its
// copies, which other CTAs hide.  Measured on the line above (ms of both
// kernels): double with 64 columns 5.64 / 4.88 / 5.08 for 2 / 3 / 4, with 32
// columns 4.53 / 3.83 / 3.62, float 21.3 / 18.0 / 16.6.
template <typename T, int NC>
constexpr int kSmallCtas = sizeof(T) > 8 ? 1 : (sizeof(T) == 8 && NC == 64 ? 3 : 4);

// what both kernels are launched with
struct SmallShape {
  int w, nb;    // largest supernode of the launch
  int early;    // 1: nothing the predecessor still runs writes the factors
  int wide;     // 1: rows of the right-hand sides are 16-byte aligned
};

template <typename T, int NC>
__global__ void __launch_bounds__(kThreads, kSmallCtas<T, NC>)
k_fwd_small(SolveArgs<T> g, SmallShape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SmallPlaces<T, NC> at(sh.w, sh.nb);
  T* Dv = reinterpret_cast<T*>(smem_raw);
  T* Lt = reinterpret_cast<T*>(smem_raw) + at.lt;
  T* Bt = reinterpret_cast<T*>(smem_raw) + at.bt;
  int32_t* rows_s = reinterpret_cast<int32_t*>(reinterpret_cast<T*>(smem_raw) + at.rows);
  // the right-hand-side chunks of a task are adjacent CTAs (its L block
  // is then read from HBM once and from L2 by the other chunks)
  const int s = g.tasks[blockIdx.x / g.nchunk].s;
  const int b = blockIdx.y;
  const int j0 = (blockIdx.x % g.nchunk) * NC;
  const int rc = min(NC, g.k - j0);
  const DevSym& S = g.S;
  const int N = S.front_n[s], first = S.sn_first[s];
  const int w = S.sn_first[s + 1] - first, w4 = (w + 3) & ~3;
  const T* F = g.fronts + int64_t(b) * g.front_stride + S.front_off[s];
  const T* Di = g.dinv + b * g.dinv_stride + g.dinv_off[s];
  const int32_t* rows = S.rows + S.rows_ptr[s];
  T* A = g.A + int64_t(b) * g.n * g.k;
  T* Bo = g.B + int64_t(b) * g.n * g.k;
  const bool wide = sh.wide != 0;
  for (int i = threadIdx.x; i < min(kSmallRows, N - w); i += kThreads) rows_s[i] = rows[w + i];
  if (sh.early) small_load_cols(Dv, at.ldd, Di, w, w, w);
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  if (ir_skip(g.skip)) {
    small_commit();
    small_wait<0>();
    return;
  }
  small_load_rhs<T, NC>(Bt, A, g.k, j0, rc, w, wide, [&](int r) { return first + r; });
  if (!sh.early) small_load_cols(Dv, at.ldd, Di, w, w, w);
  small_commit();
  small_wait<0>();
  __syncthreads();
  bool any = false;
  for (int q = threadIdx.x; q < w * NC; q += kThreads) {
    const T v = Bt[q / NC * (NC + 4) + q % NC];
    any = any || !is_zero(v);
  }
  if (!__syncthreads_or(any)) {
    for (int q = threadIdx.x; q < w * NC; q += kThreads)
      if (q % NC < rc) Bo[int64_t(first + q / NC) * g.k + j0 + q % NC] = T(0);
    return;
  }
  if (N > w) small_load_cols(Lt, at.ldl, F + w, N, min(kPanel, N - w), w);
  small_commit();
  SmallTile<T, NC> acc;
  acc.zero();
  acc.template mul<false>(Dv, at.ldd, Bt, w4, w, rc);
  __syncthreads();   // b is read: y takes its place
  acc.each(w, [&](int r, int j, T& v) {
    if (r < w) {
      Bt[r * (NC + 4) + j] = v;
      if (j < rc) Bo[int64_t(first + r) * g.k + j0 + j] = v;
    }
  });
  for (int r0 = w; r0 < N; r0 += kPanel) {
    const int nr = min(kPanel, N - r0);
    if (r0 > w) {
      __syncthreads();   // the tile before is read
      if ((r0 - w) % kSmallRows == 0)
        for (int i = threadIdx.x; i < min(kSmallRows, N - r0); i += kThreads)
          rows_s[i] = rows[r0 + i];
      small_load_cols(Lt, at.ldl, F + r0, N, nr, w);
      small_commit();
    }
    small_wait<0>();
    __syncthreads();
    acc.zero();
    acc.template mul<false>(Lt, at.ldl, Bt, w4, nr, rc);
    const int32_t* rs = rows_s + (r0 - w) % kSmallRows;
    acc.each(nr, [&](int r, int j, T& v) {
      if (r < nr && j < rc) atomicAdd(A + int64_t(rs[r]) * g.k + j0 + j, -v);
    });
  }
}

template <typename T, int NC>
__global__ void __launch_bounds__(kThreads, kSmallCtas<T, NC>)
k_bwd_small(SolveArgs<T> g, SmallShape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SmallPlaces<T, NC> at(sh.w, sh.nb);
  T* Dv = reinterpret_cast<T*>(smem_raw);
  T* Lt = reinterpret_cast<T*>(smem_raw) + at.lt;
  T* Bt = reinterpret_cast<T*>(smem_raw) + at.bt;
  int32_t* rows_s = reinterpret_cast<int32_t*>(reinterpret_cast<T*>(smem_raw) + at.rows);
  const int s = g.tasks[blockIdx.x / g.nchunk].s;
  const int b = blockIdx.y;
  const int j0 = (blockIdx.x % g.nchunk) * NC;
  const int rc = min(NC, g.k - j0);
  const DevSym& S = g.S;
  const int N = S.front_n[s], first = S.sn_first[s];
  const int w = S.sn_first[s + 1] - first, w4 = (w + 3) & ~3;
  const T* F = g.fronts + int64_t(b) * g.front_stride + S.front_off[s];
  const T* Di = g.dinv + b * g.dinv_stride + g.dinv_off[s];
  const int32_t* rows = S.rows + S.rows_ptr[s];
  T* A = g.A + int64_t(b) * g.n * g.k;
  const T* Bo = g.B + int64_t(b) * g.n * g.k;
  const bool wide = sh.wide != 0;
  auto factors = [&]() {
    if (N > w) small_load_cols(Lt, at.ldl, F + w, N, min(kPanel, N - w), w);
    small_load_cols(Dv, at.ldd, Di, w, w, w);
  };
  for (int i = threadIdx.x; i < min(kSmallRows, N - w); i += kThreads) rows_s[i] = rows[w + i];
  __syncthreads();
  if (sh.early) factors();
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  if (ir_skip(g.skip)) {
    small_commit();
    small_wait<0>();
    return;
  }
  SmallTile<T, NC> y, acc;
  y.each(w, [&](int r, int j, T& v) {
    v = r < w && j < rc ? Bo[int64_t(first + r) * g.k + j0 + j] : T(0);
  });
  acc.zero();
  for (int r0 = w; r0 < N; r0 += kPanel) {
    const int nr = min(kPanel, N - r0);
    if (r0 > w) {
      __syncthreads();   // the tile before is read
      if ((r0 - w) % kSmallRows == 0) {
        for (int i = threadIdx.x; i < min(kSmallRows, N - r0); i += kThreads)
          rows_s[i] = rows[r0 + i];
        __syncthreads();
      }
      small_load_cols(Lt, at.ldl, F + r0, N, nr, w);
    }
    const int32_t* rs = rows_s + (r0 - w) % kSmallRows;
    small_load_rhs<T, NC>(Bt, A, g.k, j0, rc, nr, wide, [&](int r) { return rs[r]; });
    if (r0 == w && !sh.early) factors();
    small_commit();
    small_wait<0>();
    __syncthreads();
    acc.template mul<true>(Lt, at.ldl, Bt, (nr + 3) & ~3, w, rc);
  }
  if (N == w && !sh.early) factors();
  small_commit();
  small_wait<0>();
  __syncthreads();   // x_B is read: y - L_B^T x_B takes its place
  {
    constexpr int n = sizeof(y.a) / sizeof(T);
    T* yp = reinterpret_cast<T*>(&y.a);
    const T* ap = reinterpret_cast<const T*>(&acc.a);
#pragma unroll
    for (int i = 0; i < n; ++i) yp[i] -= ap[i];
  }
  y.each(w4, [&](int r, int j, T& v) {
    if (r < w4) Bt[r * (NC + 4) + j] = r < w ? v : T(0);
  });
  __syncthreads();
  acc.zero();
  acc.template mul<true>(Dv, at.ldd, Bt, w4, w, rc);
  acc.each(w, [&](int r, int j, T& v) {
    if (r < w && j < rc) A[int64_t(first + r) * g.k + j0 + j] = v;
  });
}

}  // namespace
}  // namespace dct
