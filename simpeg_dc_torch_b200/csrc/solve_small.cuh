// Substitution with the supernodes of one panel (ns <= 64): one CTA per
// supernode, system and one or more chunks of NC right-hand sides.
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
//   - in launches of many CTAs one goes through several chunks of right-hand
//     sides with the factors that it copied;
//   - D^{-1} is lower triangular, and its products leave the other half out;
//   - the next launch of a pass starts early (programmatic dependent launch)
//     and copies its factors, which no launch of the pass writes, before it
//     waits for the predecessor's right-hand sides;
//   - a forward CTA whose right-hand sides are all zero writes y = 0 and is
//     done.  The sources and the adjoint sources of a survey are a few
//     electrodes, so most supernodes of the lower levels have none below them
//     (the test costs a dense right-hand side nothing: the tile has to arrive
//     before the product anyway).
// Measured on a B200, 56,525-node line, 12 systems, 186 sources, the two solves
// of an evaluation and gradient: 4.2 ms in double and 8.9 in float (which
// refines: three solves more) against 11.08 and 22.4 with 64-column register
// tiles loaded through registers, a CTA per chunk and no test for zeros.
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
// `cols` columns of the tile need be right.  TRI: A is zero for k > m ([k][m])
// or k < m ([m][k]) and those columns are left out.  each_run(rows, f) visits
// this thread's runs f(row, column, values[W]) of W columns in the first `rows`
// rows, rounded up, each(rows, f) their entries.
//
// The strided form: rows ag, ag + AG, .. and columns jg, jg + JG, .. of a
// thread, so that neighbours read and write neighbouring elements.
template <typename T, int NC>
struct StridedTile {
  using Elem = T;
  static constexpr int JG = NC >= 16 ? 16 : 8, AG = kThreads / JG, P = 64 / AG, Q = NC / JG;
  static constexpr int G = AG, W = 1;
  T a[P][Q];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int q = 0; q < Q; ++q) a[p][q] = T(0);
  }
  // row groups P0 .. P1 - 1 over the columns k0 .. k1 - 1
  template <bool MK, int P0, int P1>
  __device__ __forceinline__ void run(const T* __restrict__ A, int la, const T* __restrict__ B,
                                      int k0, int k1) {
    const int jg = threadIdx.x % JG, ag = threadIdx.x / JG;
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      T x[P1], y[Q];
#pragma unroll
      for (int p = P0; p < P1; ++p)
        x[p] = MK ? A[(ag + AG * p) * la + k] : A[k * la + ag + AG * p];
#pragma unroll
      for (int q = 0; q < Q; ++q) y[q] = B[k * (NC + 4) + jg + JG * q];
#pragma unroll
      for (int p = P0; p < P1; ++p)
#pragma unroll
        for (int q = 0; q < Q; ++q) a[p][q] += x[p] * y[q];
    }
  }
  template <bool MK, bool TRI, int NP, int I = 0>
  __device__ __forceinline__ void mul_np(const T* A, int la, const T* B, int K) {
    if constexpr (!TRI) {
      run<MK, 0, NP>(A, la, B, 0, K);
    } else if constexpr (I < NP) {
      const int k1 = I + 1 < NP ? min(K, AG * (I + 1)) : K;
      run<MK, MK ? 0 : I, MK ? I + 1 : NP>(A, la, B, min(K, AG * I), k1);
      mul_np<MK, TRI, NP, I + 1>(A, la, B, K);
    }
  }
  template <bool MK, bool TRI = false>
  __device__ __forceinline__ void mul(const T* A, int la, const T* B, int K, int rows, int) {
    const int np = (rows + AG - 1) / AG;
    if (np >= P) return mul_np<MK, TRI, P>(A, la, B, K);
    if constexpr (P > 1)
      if (np == 1) return mul_np<MK, TRI, 1>(A, la, B, K);
    if constexpr (P > 2) {
      if (np == 2) return mul_np<MK, TRI, 2>(A, la, B, K);
      mul_np<MK, TRI, 3>(A, la, B, K);
    }
  }
  template <typename Fn>
  __device__ __forceinline__ void each_run(int rows, Fn&& f) {
    const int jg = threadIdx.x % JG, ag = threadIdx.x / JG;
#pragma unroll
    for (int p = 0; p < P; ++p)
      if (AG * p < rows)
#pragma unroll
        for (int q = 0; q < Q; ++q)
          f(ag + AG * p, jg + JG * q, reinterpret_cast<T(&)[1]>(a[p][q]));
  }
  template <typename Fn>
  __device__ __forceinline__ void each(int rows, Fn&& f) {
    each_run(rows, [&](int r, int j, Elem (&v)[W]) {
#pragma unroll
      for (int h = 0; h < W; ++h) f(r, j + h, v[h]);
    });
  }
};

// complex
template <typename T, int NC>
struct SmallTile : StridedTile<T, NC> {};

// N elements at a multiple of their size
template <int N>
__device__ __forceinline__ void small_vec(float (&v)[N], const float* p) {
  if constexpr (N == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else if constexpr (N == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x, v[1] = t.y;
  } else {
    v[0] = *p;
  }
}

// float: P neighbouring rows and Q neighbouring columns of a thread, eight rows
// of a warp.  What bounds the product is shared memory: read in runs, a step
// of 16 products takes 3 wavefronts instead of 8.
template <int NC>
struct SmallTile<float, NC> {
  using Elem = float;
  static constexpr int JG = NC >= 16 ? 16 : 8, AG = kThreads / JG, P = 64 / AG, Q = NC / JG;
  static constexpr int G = 8, W = Q;
  static_assert(P * 32 / JG == 8, "a warp has eight rows");
  float a[P][Q];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int q = 0; q < Q; ++q) a[p][q] = 0.f;
  }
  template <bool MK, bool TRI = false>
  __device__ __forceinline__ void mul(const float* __restrict__ A, int la,
                                      const float* __restrict__ B, int K, int rows, int) {
    const int jg = threadIdx.x % JG, ag = threadIdx.x / JG, r8 = threadIdx.x / 32 * 8;
    if (r8 >= rows) return;
    const int k0 = TRI && MK ? r8 : 0, k1 = TRI && !MK ? min(K, r8 + 8) : K;
    const float* pa = A + (MK ? P * ag * la : P * ag);
    const float* pb = B + jg * Q;
    if constexpr (MK) {
#pragma unroll 1
      for (int k = k0; k < k1; k += 4) {
        float x[P][4], y[Q];
#pragma unroll
        for (int p = 0; p < P; ++p) small_vec<4>(x[p], pa + p * la + k);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          small_vec<Q>(y, pb + (k + h) * (NC + 4));
#pragma unroll
          for (int p = 0; p < P; ++p)
#pragma unroll
            for (int q = 0; q < Q; ++q) a[p][q] += x[p][h] * y[q];
        }
      }
    } else {
#pragma unroll 4
      for (int k = k0; k < k1; ++k) {
        float x[P], y[Q];
        small_vec<P>(x, pa + k * la);
        small_vec<Q>(y, pb + k * (NC + 4));
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
          for (int q = 0; q < Q; ++q) a[p][q] += x[p] * y[q];
      }
    }
  }
  template <typename Fn>
  __device__ __forceinline__ void each_run(int rows, Fn&& f) {
    const int jg = threadIdx.x % JG, ag = threadIdx.x / JG;
    if (int(threadIdx.x / 32 * 8) >= rows) return;
#pragma unroll
    for (int p = 0; p < P; ++p) f(P * ag + p, jg * Q, a[p]);
  }
  template <typename Fn>
  __device__ __forceinline__ void each(int rows, Fn&& f) {
    each_run(rows, [&](int r, int j, Elem (&v)[W]) {
#pragma unroll
      for (int h = 0; h < W; ++h) f(r, j + h, v[h]);
    });
  }
};

// double: 8 x 8 tensor-core fragments; the row fragments are dealt out to the
// warps in turn and back again, so that a supernode of few rows still occupies
// all of them and the triangular products are even
template <int NC>
struct SmallTile<double, NC> {
  using Elem = double;
  static constexpr int WM = NC == 64 ? 2 : (NC == 32 ? 4 : 8), WN = 8 / WM;
  static constexpr int MF = 8 / WM, NF = NC / 8 / WN, G = 8, W = 2;
  double a[MF][NF][2];
  // first row of fragment p of this warp
  static __device__ __forceinline__ int row(int p) {
    const int wm = (threadIdx.x >> 5) % WM;
    return 8 * (WM * p + (p % 2 ? WM - 1 - wm : wm));
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < MF; ++p)
#pragma unroll
      for (int q = 0; q < NF; ++q) a[p][q][0] = a[p][q][1] = 0.0;
  }
  template <bool MK, int P0, int P1>
  __device__ __forceinline__ void run(const double* __restrict__ A, int la,
                                      const double* __restrict__ B, int k0, int k1) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // fragments p = 0, 2, .. and p = 1, 3, .. are 16 WM rows apart each
    const int r0 = row(0) + g, r1 = MF > 1 ? row(1) - 8 * WM + g : 0;
    const double* p0 = MK ? A + r0 * la + k0 + t : A + (k0 + t) * la + r0;
    const double* p1 = MK ? A + r1 * la + k0 + t : A + (k0 + t) * la + r1;
    const int sm = MK ? 8 * WM * la : 8 * WM;
    const double* pb = B + (k0 + t) * (NC + 4) + 8 * NF * (warp / WM) + g;
    const int sa = MK ? 4 : 4 * la;
#pragma unroll 4
    for (int k = k0; k < k1; k += 4, p0 += sa, p1 += sa, pb += 4 * (NC + 4)) {
      double x[P1], y[NF];
#pragma unroll
      for (int p = P0; p < P1; ++p) x[p] = (p % 2 ? p1 : p0)[p * sm];
#pragma unroll
      for (int q = 0; q < NF; ++q) y[q] = pb[8 * q];
#pragma unroll
      for (int p = P0; p < P1; ++p)
#pragma unroll
        for (int q = 0; q < NF; ++q) dmma(a[p][q], x[p], y[q]);
    }
  }
  template <bool MK, bool TRI, int NP, int I = 0>
  __device__ __forceinline__ void mul_np(const double* A, int la, const double* B, int K) {
    if constexpr (!TRI) {
      run<MK, 0, NP>(A, la, B, 0, K);
    } else if constexpr (I < NP) {
      if constexpr (MK)
        run<MK, 0, I + 1>(A, la, B, row(I), I + 1 < NP ? row(I + 1) : K);
      else
        run<MK, I, NP>(A, la, B, I > 0 ? row(I - 1) + 8 : 0, min(K, row(I) + 8));
      mul_np<MK, TRI, NP, I + 1>(A, la, B, K);
    }
  }
  template <bool MK, bool TRI = false>
  __device__ __forceinline__ void mul(const double* A, int la, const double* B, int K, int rows,
                                      int cols) {
    if (row(0) >= rows || 8 * NF * int((threadIdx.x >> 5) / WM) >= cols) return;
    if (row(MF - 1) < rows) return mul_np<MK, TRI, MF>(A, la, B, K);
    if constexpr (MF > 2) {
      if (row(2) < rows) return mul_np<MK, TRI, 3>(A, la, B, K);
      if (row(1) < rows) return mul_np<MK, TRI, 2>(A, la, B, K);
    }
    if constexpr (MF > 1) mul_np<MK, TRI, 1>(A, la, B, K);
  }
  template <typename Fn>
  __device__ __forceinline__ void each_run(int rows, Fn&& f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int p = 0; p < MF; ++p)
      if (row(p) < rows)
#pragma unroll
        for (int q = 0; q < NF; ++q)
          f(row(p) + g, 8 * (NF * (warp / WM) + q) + 2 * t, a[p][q]);
  }
  template <typename Fn>
  __device__ __forceinline__ void each(int rows, Fn&& f) {
    each_run(rows, [&](int r, int j, Elem (&v)[W]) {
#pragma unroll
      for (int h = 0; h < W; ++h) f(r, j + h, v[h]);
    });
  }
};

// W neighbouring right-hand sides of a row, as many as lie before `left`; wide:
// in one access (then left is none or all of them)
template <typename T, int W>
__device__ __forceinline__ void small_get(T (&v)[W], const T* p, int left, bool wide) {
  struct alignas(W * sizeof(T)) Run { T v[W]; };
  if (W > 1 && wide) {
    if (left > 0) {
      const Run t = *reinterpret_cast<const Run*>(p);
#pragma unroll
      for (int h = 0; h < W; ++h) v[h] = t.v[h];
    } else {
#pragma unroll
      for (int h = 0; h < W; ++h) v[h] = T(0);
    }
  } else {
#pragma unroll
    for (int h = 0; h < W; ++h) v[h] = h < left ? p[h] : T(0);
  }
}
template <typename T, int W>
__device__ __forceinline__ void small_put(T* p, const T (&v)[W], int left, bool wide) {
  struct alignas(W * sizeof(T)) Run { T v[W]; };
  if (W > 1 && wide) {
    if (left > 0) {
      Run t;
#pragma unroll
      for (int h = 0; h < W; ++h) t.v[h] = v[h];
      *reinterpret_cast<Run*>(p) = t;
    }
  } else {
#pragma unroll
    for (int h = 0; h < W; ++h)
      if (h < left) p[h] = v[h];
  }
}
// p -= v; four floats in one reduction
template <typename T, int W>
__device__ __forceinline__ void small_sub(T* p, const T (&v)[W], int left, bool wide) {
  if constexpr (sizeof(T) == 4 && W == 4) {
    if (wide) {
      if (left > 0)
        atomicAdd(reinterpret_cast<float4*>(p), make_float4(-v[0], -v[1], -v[2], -v[3]));
      return;
    }
  }
#pragma unroll
  for (int h = 0; h < W; ++h)
    if (h < left) atomicAdd(p + h, -v[h]);
}

// shared-memory places (in elements) of a launch whose supernodes have at
// most w columns and nb boundary rows: D^{-1}, a tile of L_B, the right-hand
// sides that arrive (xt: in rows of them) and the products that leave for the
// other product (yt).  A CTA of one chunk has both in one place.
constexpr int kSmallRows = 1024;   // row indices kept at a time
template <typename T, int NC>
struct SmallPlaces {
  int ldd, ldl, lt, xt, yt, rows;
  __host__ __device__ SmallPlaces(int w, int nb, int in, bool apart) {
    const int r = nb < kPanel ? nb : kPanel;
    // the [m][k] products read whole row groups of the tile's threads
    constexpr int G = SmallTile<T, NC>::G;
    const int wr = (w + G - 1) / G * G;
    ldd = ((w + 7) & ~7) + 4;      // 4 modulo 8, and room for the row padding
    ldl = ((r + 7) & ~7) + 4;
    lt = wr * ldd;
    xt = lt + wr * ldl;
    const int x = ((in + 3) & ~3) * (NC + 4), y = ((w + 3) & ~3) * (NC + 4);
    yt = apart ? xt + x : xt;
    rows = apart ? yt + y : xt + (x > y ? x : y);
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
// copies, which other CTAs hide.  Measured (ms of both kernels, without the
// loop over chunks): double with 64 columns on the line above 5.64 / 4.88 /
// 5.08 for 2 / 3 / 4, with 32 columns on ten lines of 72 sources 4.53 / 3.83 /
// 3.62, float 21.3 / 18.0 / 16.6.
template <typename T, int NC>
constexpr int kSmallCtas = sizeof(T) > 8 ? 1 : (sizeof(T) == 8 && NC == 64 ? 3 : 4);

// whether a CTA can go through several chunks (LOOP; the kernels of one chunk
// are compiled without the loop, which spills a few registers).  Double tiles of 64 columns
// would spill the next chunk's rows, and the second set of a complex CTA's
// right-hand sides does not fit its shared memory.
template <typename T, int NC>
constexpr bool kSmallLoop = sizeof(T) == 4 ? NC >= 32 : (sizeof(T) == 8 && NC == 32);

// Right-hand sides per chunk: the fewest columns that hold k, or chunks of 64
// or 32.  Double supernodes of at most one tile of boundary rows take 32 where
// 64 leave several chunks, which one CTA then goes through (measured, bwd + fwd
// of a pass: 4.23 ms against 4.67 on the line above), and where three CTAs of
// 64 do not share an SM (leaves of 63 columns, ten lines of 72 sources: 3.4
// against 4.5 ms); one chunk of 64 beats two of 32 otherwise (38 sources, leaves
// of 54 columns: 2.42 against 2.78 ms).  With more boundary rows each chunk reads
// L_B again and 64 are better (2.5 against 3.1 ms on the 269,001-node benchmark)
// unless they leave a fifth of the columns empty.
template <typename T>
int small_columns(int k, int w, int nb) {
  if (k <= 32) return k <= 8 ? 8 : (k <= 16 ? 16 : 32);
  constexpr size_t third = 75 * 1024;   // of an SM's shared memory
  if (sizeof(T) == 8 && nb <= kPanel &&
      (k > 64 || SmallPlaces<T, 64>(w, nb, w, false).bytes(nb) > third))
    return 32;
  const int c64 = (k + 63) / 64 * 64, c32 = (k + 31) / 32 * 32;
  return 5 * c32 <= 4 * c64 ? 32 : 64;
}

// Chunks that a CTA goes through: all of them in launches of many CTAs, so that
// the factors are copied once and the next chunk's right-hand sides arrive
// during the products of this one; fewer where kSmallLaunch CTAs would not be
// left (888 to 2,000 measured alike), one where a chunk needs several tiles
// of L_B, which are copied again for each.
constexpr int64_t kSmallLaunch = 2048;
template <typename T, int NC>
int small_chunks(int64_t tasks, int nb, int nchunk) {
  if (!kSmallLoop<T, NC> || nb > kPanel) return 1;
  const int64_t most = (kSmallLaunch + tasks - 1) / tasks;
  const int ngroup = most < nchunk ? static_cast<int>(most) : nchunk;
  return (nchunk + ngroup - 1) / ngroup;
}

// what both kernels are launched with
struct SmallShape {
  int w, nb;    // largest supernode of the launch
  int early;    // 1: nothing the predecessor still runs writes the factors
  int wide;     // 1: rows of the right-hand sides are 16-byte aligned
  int chunks;   // chunks of NC right-hand sides that a CTA goes through
};

template <typename T, int NC, bool LOOP>
__global__ void __launch_bounds__(kThreads, kSmallCtas<T, NC>)
k_fwd_small(SolveArgs<T> g, SmallShape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int W = SmallTile<T, NC>::W;
  constexpr bool apart = LOOP;
  const SmallPlaces<T, NC> at(sh.w, sh.nb, sh.w, apart);
  T* Dv = reinterpret_cast<T*>(smem_raw);
  T* Lt = Dv + at.lt;
  T* Xt = Dv + at.xt;
  T* Yt = Dv + at.yt;
  int32_t* rows_s = reinterpret_cast<int32_t*>(Dv + at.rows);
  // the groups of chunks of a task are adjacent CTAs (its L block is then
  // read from HBM once and from L2 by the others)
  const int chunks = LOOP ? sh.chunks : 1, ngroup = (g.nchunk + chunks - 1) / chunks;
  const int s = g.tasks[blockIdx.x / ngroup].s;
  const int b = blockIdx.y;
  const int jb = blockIdx.x % ngroup * chunks * NC, je = min(g.k, jb + chunks * NC);
  const DevSym& S = g.S;
  const int N = S.front_n[s], first = S.sn_first[s];
  const int w = S.sn_first[s + 1] - first, w4 = (w + 3) & ~3;
  const T* F = g.fronts + int64_t(b) * g.front_stride + S.front_off[s];
  const T* Di = g.dinv + b * g.dinv_stride + g.dinv_off[s];
  const int32_t* rows = S.rows + S.rows_ptr[s];
  T* A = g.A + int64_t(b) * g.n * g.k;
  T* Bo = g.B + int64_t(b) * g.n * g.k;
  const bool wide = sh.wide != 0;
  const T* src = g.b != nullptr ? g.b + b * g.bstride : A;
  auto load_b = [&](int j0) {
    small_load_rhs<T, NC>(Xt, src, g.k, j0, min(NC, je - j0), w, wide,
                          [&](int r) { return first + r; });
  };
  for (int i = threadIdx.x; i < min(kSmallRows, N - w); i += kThreads) rows_s[i] = rows[w + i];
  if (sh.early) small_load_cols(Dv, at.ldd, Di, w, w, w);
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  if (ir_skip(g.skip)) {
    small_commit();
    small_wait<0>();
    return;
  }
  load_b(jb);
  if (!sh.early) small_load_cols(Dv, at.ldd, Di, w, w, w);
  small_commit();
  // a run of the rows that the other product reads, zeros beyond w
  auto rows_up = [&](int r, int j, T (&v)[W]) {
    if (r < w4) {
      if (r >= w)
#pragma unroll
        for (int h = 0; h < W; ++h) v[h] = T(0);
      small_put<T, W>(Yt + r * (NC + 4) + j, v, W, true);
    }
  };
  bool held = false;   // Lt is the first tile of L_B
  for (int j0 = jb; j0 < je; j0 += NC) {
    const int rc = min(NC, je - j0);
    const bool more = LOOP && j0 + NC < je;
    small_wait<0>();
    __syncthreads();   // b is here; the products of the chunk before are done
    bool any = false;
    for (int q = threadIdx.x; q < w * NC; q += kThreads) {
      const T v = Xt[q / NC * (NC + 4) + q % NC];
      any = any || !is_zero(v);
    }
    if (!__syncthreads_or(any)) {
      if (more) load_b(j0 + NC);
      small_commit();
      for (int q = threadIdx.x; q < w * NC; q += kThreads)
        if (q % NC < rc) Bo[int64_t(first + q / NC) * g.k + j0 + q % NC] = T(0);
      continue;
    }
    if (N > w && !held) small_load_cols(Lt, at.ldl, F + w, N, min(kPanel, N - w), w);
    held = N - w <= kPanel;
    small_commit();
    SmallTile<T, NC> acc;
    acc.zero();
    acc.template mul<false, true>(Dv, at.ldd, Xt, w4, w, rc);
    if (!apart) __syncthreads();   // b is read: y takes its place
    acc.each_run(w4, [&](int r, int j, T (&v)[W]) {
      if (r < w) small_put<T, W>(Bo + int64_t(first + r) * g.k + j0 + j, v, rc - j, wide);
      rows_up(r, j, v);
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
      if (r0 == w && more) {   // b is read
        load_b(j0 + NC);
        small_commit();
      }
      acc.zero();
      acc.template mul<false>(Lt, at.ldl, Yt, w4, nr, rc);
      const int32_t* rs = rows_s + (r0 - w) % kSmallRows;
      acc.each_run(nr, [&](int r, int j, T (&v)[W]) {
        if (r < nr) small_sub<T, W>(A + int64_t(rs[r]) * g.k + j0 + j, v, rc - j, wide);
      });
    }
    if (N == w && more) {
      __syncthreads();   // b is read
      load_b(j0 + NC);
      small_commit();
    }
    if (!LOOP) break;
  }
  small_wait<0>();
}

template <typename T, int NC, bool LOOP>
__global__ void __launch_bounds__(kThreads, kSmallCtas<T, NC>)
k_bwd_small(SolveArgs<T> g, SmallShape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int W = SmallTile<T, NC>::W;
  constexpr bool apart = LOOP;
  const SmallPlaces<T, NC> at(sh.w, sh.nb, min(sh.nb, kPanel), apart);
  T* Dv = reinterpret_cast<T*>(smem_raw);
  T* Lt = Dv + at.lt;
  T* Xt = Dv + at.xt;
  T* Yt = Dv + at.yt;
  int32_t* rows_s = reinterpret_cast<int32_t*>(Dv + at.rows);
  const int chunks = LOOP ? sh.chunks : 1, ngroup = (g.nchunk + chunks - 1) / chunks;
  const int s = g.tasks[blockIdx.x / ngroup].s;
  const int b = blockIdx.y;
  const int jb = blockIdx.x % ngroup * chunks * NC, je = min(g.k, jb + chunks * NC);
  const DevSym& S = g.S;
  const int N = S.front_n[s], first = S.sn_first[s];
  const int w = S.sn_first[s + 1] - first, w4 = (w + 3) & ~3;
  const T* F = g.fronts + int64_t(b) * g.front_stride + S.front_off[s];
  const T* Di = g.dinv + b * g.dinv_stride + g.dinv_off[s];
  const int32_t* rows = S.rows + S.rows_ptr[s];
  T* A = g.A + int64_t(b) * g.n * g.k;
  const T* Bo = g.B + int64_t(b) * g.n * g.k;
  const bool wide = sh.wide != 0;
  auto load_l = [&](int r0) {
    small_load_cols(Lt, at.ldl, F + r0, N, min(kPanel, N - r0), w);
  };
  auto load_x = [&](int r0, int j0) {
    const int32_t* rs = rows_s + (r0 - w) % kSmallRows;
    small_load_rhs<T, NC>(Xt, A, g.k, j0, min(NC, je - j0), min(kPanel, N - r0), wide,
                          [&](int r) { return rs[r]; });
  };
  SmallTile<T, NC> y, acc;
  auto load_y = [&](int j0) {
    y.each_run(w, [&](int r, int j, T (&v)[W]) {
      small_get<T, W>(v, Bo + int64_t(first + r) * g.k + j0 + j, r < w ? je - j0 - j : 0, wide);
    });
  };
  auto factors = [&]() {
    if (N > w) load_l(w);
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
  load_y(jb);
  if (N > w) load_x(w, jb);
  if (!sh.early) factors();
  small_commit();
  for (int j0 = jb; j0 < je; j0 += NC) {
    const int rc = min(NC, je - j0);
    const bool more = LOOP && j0 + NC < je;
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
        load_l(r0);
        load_x(r0, j0);
        small_commit();
      }
      small_wait<0>();
      __syncthreads();   // (and the products of the chunk before are done)
      acc.template mul<true>(Lt, at.ldl, Xt, (nr + 3) & ~3, w, rc);
    }
    if (N == w) small_wait<0>();
    if (N == w || !apart) __syncthreads();   // x_B is read: y - L_B^T x_B takes its place
    {
      constexpr int n = sizeof(y.a) / sizeof(T);
      T* yp = reinterpret_cast<T*>(&y.a);
      const T* ap = reinterpret_cast<const T*>(&acc.a);
#pragma unroll
      for (int i = 0; i < n; ++i) yp[i] -= ap[i];
    }
    y.each_run(w4, [&](int r, int j, T (&v)[W]) {
      if (r >= w)
#pragma unroll
        for (int h = 0; h < W; ++h) v[h] = T(0);
      if (r < w4) small_put<T, W>(Yt + r * (NC + 4) + j, v, W, true);
    });
    if (more) load_y(j0 + NC);
    __syncthreads();
    if (more && N > w) {   // x_B is read
      if (N - w > kPanel) load_l(w);
      load_x(w, j0 + NC);
      small_commit();
    }
    acc.zero();
    acc.template mul<true, true>(Dv, at.ldd, Yt, w4, w, rc);
    acc.each_run(w, [&](int r, int j, T (&v)[W]) {
      if (r < w) small_put<T, W>(A + int64_t(first + r) * g.k + j0 + j, v, rc - j, wide);
    });
    if (!LOOP) break;
  }
}

}  // namespace
}  // namespace dct
