// Fronts of order N <= the single-CTA limit: one CTA assembles the front in
// shared memory, eliminates its ns pivot columns, forms the inverses of the
// diagonal blocks of its 64-column panels and leaves the Schur complement.
//
// What bounds it is the chain through the pivots, so the elimination is
// blocked by 16 columns, with two barriers per block instead of two per
// pivot:
//   (a) warp 0 factors the 16 x 16 diagonal block in registers, while the
//       others apply the block before to the remaining columns of the panel
//       (warp 0 did the diagonal block's own tile first) and complete a row
//       of the panel's inverse X = D^{-1},
//         X_ij = -X_ii sum_k L_ik X_kj;
//   (b) the rows below it, one thread per row, by forward substitution
//       against that block (its entries are shared-memory broadcasts), while
//       the last warp forms the block's inverse X_ii;
// and after the last block of a panel the rest of the front takes the
// panel's update at once (16 x 16 tiles, tensor cores for double).
// X is kept transposed in the unused upper triangle of the panel's diagonal
// block (its diagonal in xd), so it costs no shared memory, and a separate
// pass over the factors to invert their diagonal blocks is not needed.
//
// Measured on a B200 in double: the 2,047 fronts x 12 systems of a 56,525-node
// line 1.25 ms, where an elimination pivot by pivot took 3.64 ms and the
// inverses of the diagonal blocks in a launch of their own 1.88 ms; the 255
// fronts x 11 systems of a 7,381-node line, all latency, 0.27 ms (0.71 + 0.23).
#pragma once
#include <cuda_runtime.h>

#include "dct_internal.h"
#include "dmma.cuh"
#include "factor_diag.cuh"

namespace dct {
namespace {

template <typename T>
__device__ __forceinline__ T load_val(const void* p, int dtype, int64_t i) {
  if constexpr (sizeof(T) == sizeof(cplx)) {
    if (dtype == DCT_C128) return static_cast<const cplx*>(p)[i];
  }
  return dtype == DCT_F64 ? T(static_cast<const double*>(p)[i])
                          : T(static_cast<const float*>(p)[i]);
}

// leading dimension of a front in shared memory: 4 modulo 8 for the double
// tensor-core fragments, packed otherwise
template <typename T>
__host__ __device__ constexpr int small_ld(int N) {
  return sizeof(T) == 8 ? N + ((12 - (N & 7)) & 7) : N;
}
// the front, its inverse diagonal (and what the shifted loops read past it) and
// two row maps
template <typename T>
__host__ __device__ constexpr size_t small_smem(int N) {
  return sizeof(T) * (size_t(small_ld<T>(N)) * N + N + 16) + 2 * sizeof(int32_t) * N;
}
// Threads per CTA: the launch's fronts up to this order take 128, so that
// twice as many of them share an SM and hide one another's pivot chains.
constexpr int kSmallNarrow = 112;

// d = sqrt(p), r = 1 / d of a pivot, both correctly rounded in float and double
// at any scale.  All pivots of a block take theirs at once, one per lane, off
// the chain from pivot to pivot.
template <typename T>
__device__ __forceinline__ void pivot_root(T p, T& d, T& r) {
  d = sqrt(p);
  r = T(1) / d;
}

// entry (r, c) of the panel inverse kept transposed above the diagonal
template <typename T>
__device__ __forceinline__ T xinv(const T* F, const T* xd, int ld, int r, int c) {
  return r > c ? F[c + r * ld] : (r == c ? xd[r] : T(0));
}

// The three pieces of a block step are loops over its pivots, four unrolled:
// the registers are shifted by one column per step, v[j - 1] = v[j] - l l_j,
// so the pivot's column is always v[0].  (A 16 x 16 Cholesky on one warp, in
// cycles: rolled 3,660, by fours 2,630, unrolled 2,180 when its instructions
// are at hand, but a front fetches them once, from the L2 cache.)  The shift
// brings in columns beyond the block, which nothing reads.

// The factorization below with every pivot tested, for a block in which one
// was not good; the entries are those kept above the diagonal and in xd.
template <typename T>
__device__ __noinline__ void small_leaf_tested(T* F, T* xd, int ld, int o, int wb, int* status,
                                               int s, int b) {
  const int i = threadIdx.x & 31;
  if (i < wb) {
    for (int q = 0; q < i; ++q) F[(o + i) + (o + q) * ld] = F[(o + q) + (o + i) * ld];
    F[(o + i) + (o + i) * ld] = xd[o + i];
  }
  __syncwarp();
  for (int k = 0; k < wb; ++k) {
    T piv = F[(o + k) + (o + k) * ld];
    if (!good_pivot(piv)) {
      piv = T(1);
      if (i == 0) flag_pivot(status, s, b);
    }
    T d, r;
    pivot_root(piv, d, r);
    __syncwarp();
    if (i > k && i < wb) F[(o + i) + (o + k) * ld] *= r;
    if (i == k) {
      F[(o + k) + (o + k) * ld] = d;
      xd[o + k] = r;
    }
    __syncwarp();
    if (i < wb)
      for (int q = k + 1; q <= i; ++q)
        F[(o + i) + (o + q) * ld] -= F[(o + i) + (o + k) * ld] * F[(o + q) + (o + k) * ld];
    __syncwarp();
  }
}

// (a) Cholesky of the wb x wb block at o (wb <= 16), one warp.  The steps use
// the unscaled columns u_k, v_j -= (u_k / p_k) u_k[j], so that the chain from
// pivot to pivot holds one reciprocal and no test; columns are broadcast
// through shared memory (thirty shuffles of half a double take longer).  The
// roots of all pivots are taken at the end, one per lane, and the columns
// scaled; if a pivot was not good the block is done again, tested.
template <typename T>
__device__ __forceinline__ void small_leaf(T* F, T* xd, int ld, int o, int wb, int* status,
                                           int s, int b) {
  const int lane = threadIdx.x & 31, i = lane & 15;
  T v[16];
#pragma unroll
  for (int q = 0; q < 16; ++q)
    v[q] = (i < wb && q <= i) ? F[(o + i) + (o + q) * ld] : T(0);
  if (lane < wb) {   // kept above the diagonal, where X will be
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      if (q < i) F[(o + q) + (o + i) * ld] = v[q];
      if (q == i) xd[o + i] = v[q];
    }
  }
  T* row = F + (o + i) + o * ld;
  T own = T(1);
#pragma unroll 1
  for (int k4 = 0; k4 < wb; k4 += 4)
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int k = k4 + kk;
      const T* diag = F + o + o * ld + min(k, wb - 1) * (ld + 1);
      const T u = v[0];
      if (lane >= k && lane < wb) row[k * ld] = u;
      __syncwarp();
      const T piv = diag[0];
      T uj[16];
#pragma unroll
      for (int j = 1; j < 16; ++j) uj[j] = diag[j];
      if (i == k) own = piv;
      const T w = u * (T(1) / piv);
#pragma unroll
      for (int j = 1; j < 16; ++j) v[j - 1] = v[j] - w * uj[j];
    }
  if (__any_sync(0xffffffffu, !good_pivot(own))) {
    small_leaf_tested(F, xd, ld, o, wb, status, s, b);
    return;
  }
  T d, r;
  pivot_root(own, d, r);
  if (lane < wb) {
    row[i * ld] = d;
    xd[o + i] = r;
  }
  __syncwarp();
  if (lane < wb) {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = k < i ? row[k * ld] * xd[o + k] : T(0);
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < i) row[k * ld] = v[k];
  }
}

// inverse of the factored block at o: lane j holds column j; one warp
template <typename T>
__device__ __forceinline__ void small_leaf_inverse(T* F, const T* xd, int ld, int o, int wb) {
  const int j = threadIdx.x & 31;
  T x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = i == j ? T(1) : T(0);
#pragma unroll 1
  for (int i4 = 0; i4 < wb; i4 += 4)
#pragma unroll
    for (int ii = 0; ii < 4; ++ii) {
      const int i = i4 + ii, ic = min(i, wb - 1);
      const T* diag = F + o + o * ld + ic * (ld + 1);
      T l[16];
#pragma unroll
      for (int q = 1; q < 16; ++q) l[q] = diag[q];
      const T xi = x[0] * xd[o + ic];
#pragma unroll
      for (int q = 1; q < 16; ++q) x[q - 1] = x[q] - l[q] * xi;
      if (j < i && i < wb) F[(o + j) + (o + i) * ld] = xi;
    }
}

// (b) row r of the block column at o: v L^T = F[r, o ..], one thread
template <typename T>
__device__ __forceinline__ void small_row_solve(T* F, const T* xd, int ld, int o, int wb, int r) {
  T v[16];
  T* row = F + r + o * ld;
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = q < wb ? row[q * ld] : T(0);
#pragma unroll 1
  for (int k4 = 0; k4 < wb; k4 += 4)
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int k = k4 + kk, kc = min(k, wb - 1);
      const T* diag = F + o + o * ld + kc * (ld + 1);
      T l[16];
#pragma unroll
      for (int j = 1; j < 16; ++j) l[j] = diag[j];
      const T vk = v[0] * xd[o + kc];
#pragma unroll
      for (int j = 1; j < 16; ++j) v[j - 1] = v[j] - vk * l[j];
      if (k < wb) row[k * ld] = vk;
    }
}

// F[r, c] -= sum_{k0 <= k < k0 + kw} F[r, k] F[c, k] on the TS x TS tile at
// (r0, c0), its entries r >= c, r < N, c < cend; one warp
template <typename T>
constexpr int kSyrkTile = sizeof(T) == 4 ? 32 : 16;

// (KW: the number of columns where it is known, else 0 and kw)
template <int KW, typename T>
__device__ __forceinline__ void syrk_tile(T* F, int ld, int N, int r0, int c0, int cend, int k0,
                                          int kw) {
  if constexpr (KW > 0) kw = KW;
  const int lane = threadIdx.x & 31;
  if constexpr (sizeof(T) == 8) {
    const int g = lane >> 2, t = lane & 3;
    int ra[2], cb[2];
    double acc[2][2][2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      ra[p] = min(r0 + 8 * p + g, N - 1);
      cb[p] = min(c0 + 8 * p + g, N - 1);
#pragma unroll
      for (int q = 0; q < 2; ++q) acc[p][q][0] = acc[p][q][1] = 0.0;
    }
#pragma unroll 4
    for (int k = 0; k < kw; k += 4) {   // 16 columns' loads in flight
      const bool in = k + t < kw;
      const double* col = F + (k0 + k + t) * ld;
      double a[2], bq[2];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        a[p] = in ? col[ra[p]] : 0.0;
        bq[p] = in ? col[cb[p]] : 0.0;
      }
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q) dmma(acc[p][q], a[p], bq[q]);
    }
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = r0 + 8 * p + g, c = c0 + 8 * q + 2 * t + h;
          if (r < N && c < cend && c <= r) F[r + c * ld] -= acc[p][q][h];
        }
  } else {
    constexpr int TS = kSyrkTile<T>, P = TS / 8, Q = TS / 4;
    const int rg = lane & 7, cg = lane >> 3;
    T acc[P][Q];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int q = 0; q < Q; ++q) acc[p][q] = T(0);
    for (int k = k0; k < k0 + kw; ++k) {
      T x[P], y[Q];
#pragma unroll
      for (int p = 0; p < P; ++p) x[p] = F[min(r0 + rg + 8 * p, N - 1) + k * ld];
#pragma unroll
      for (int q = 0; q < Q; ++q) y[q] = F[min(c0 + cg + 4 * q, N - 1) + k * ld];
#pragma unroll
      for (int p = 0; p < P; ++p)
#pragma unroll
        for (int q = 0; q < Q; ++q) acc[p][q] += x[p] * y[q];
    }
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int r = r0 + rg + 8 * p, c = c0 + cg + 4 * q;
        if (r < N && c < cend && c <= r) F[r + c * ld] -= acc[p][q];
      }
  }
}

// tile (i, j), j <= i, j < ntj, of a trapezoid by its number: the triangle
// of the first ntj tile rows, then whole rows of ntj tiles
__device__ __forceinline__ void trapezoid_tile(int q, int ntj, int& i, int& j) {
  const int tri = ntj * (ntj + 1) / 2;
  if (q < tri) {
    i = int((sqrtf(8.0f * q + 1.0f) - 1.0f) * 0.5f);
    while ((i + 1) * (i + 2) / 2 <= q) ++i;
    while (i * (i + 1) / 2 > q) --i;
    j = q - i * (i + 1) / 2;
  } else {
    i = ntj + (q - tri) / ntj;
    j = (q - tri) % ntj;
  }
}
__device__ __forceinline__ int trapezoid_tiles(int nti, int ntj) {
  return ntj * (ntj + 1) / 2 + (nti - ntj) * ntj;
}

// the next tile of a phase, for a whole warp
__device__ __forceinline__ int take_tile(int* next_tile) {
  int q = 0;
  if ((threadIdx.x & 31) == 0) q = atomicAdd(next_tile, 1);
  return __shfl_sync(0xffffffffu, q, 0);
}

// X_ij of the panel inverse, 16 x 16 at (i16, j16), one warp; pend = end of
// the panel's columns.  The sum is formed in the block's own place.
template <typename T>
__device__ __forceinline__ void small_xblock(T* F, const T* xd, int ld, int i16, int j16,
                                             int pend) {
  const int lane = threadIdx.x & 31;
  if constexpr (sizeof(T) == 8) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      double acc[2][2][2];
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q) acc[p][q][0] = acc[p][q][1] = 0.0;
      const int ka = pass == 0 ? j16 : i16, ke = pass == 0 ? i16 : min(i16 + 16, pend);
#pragma unroll 4
      for (int k = ka; k < ka + (pass == 0 ? i16 - j16 : 16); k += 4) {
        const int kk = k + t;
        double a[2], bq[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const int r = i16 + 8 * p + g, c = j16 + 8 * p + g;
          const bool in = kk < ke;
          if (pass == 0) {
            a[p] = (in && r < pend) ? F[r + kk * ld] : 0.0;
            bq[p] = in ? xinv(F, xd, ld, kk, c) : 0.0;
          } else {
            a[p] = (in && r < pend) ? xinv(F, xd, ld, r, kk) : 0.0;
            bq[p] = in ? F[c + kk * ld] : 0.0;
          }
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int q = 0; q < 2; ++q) dmma(acc[p][q], a[p], bq[q]);
      }
      __syncwarp();
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = i16 + 8 * p + g, c = j16 + 8 * q + 2 * t + h;
            if (r < pend) F[c + r * ld] = pass == 0 ? acc[p][q][h] : -acc[p][q][h];
          }
      __syncwarp();
    }
  } else {
    const int r = i16 + (lane & 15), cb = j16 + (lane >> 4) * 8;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      T acc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = T(0);
      const int ka = pass == 0 ? j16 : i16, ke = pass == 0 ? i16 : min(i16 + 16, pend);
      if (r < pend)
        for (int k = ka; k < ke; ++k) {
          const T a = pass == 0 ? F[r + k * ld] : xinv(F, xd, ld, r, k);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            acc[q] += a * (pass == 0 ? xinv(F, xd, ld, k, cb + q) : F[(cb + q) + k * ld]);
        }
      __syncwarp();
      if (r < pend) {
#pragma unroll
        for (int q = 0; q < 8; ++q) F[(cb + q) + r * ld] = pass == 0 ? acc[q] : -acc[q];
      }
      __syncwarp();
    }
  }
}

// The columns c0 .. pend (one panel) of the N x N block F: factored, the rows
// below them solved, and their inverse but for its last row.  Every column
// right of the panel still lacks the panel's update.  next_tile: a word of
// shared memory, 0 when it returns.
template <typename T, int NT>
__device__ __forceinline__ void small_panel(T* F, T* xd, int ld, int N, int c0, int pend,
                                            int* next_tile, int* status, int s, int b) {
  constexpr int TS = kSyrkTile<T>, kW = NT / 32;
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int o = c0, blk = 0; o < pend; o += 16, ++blk) {
    const int wb = min(16, pend - o), nx = o + wb;
    // Columns o .. pend take the update of the block before.  Warp 0 does
    // the tile of the next diagonal block and factors that at once; the
    // others do the rest and the row of X that the block before completed.
    const int nti = (N - o + TS - 1) / TS, ntj = (pend - o + TS - 1) / TS;
    if (warp == 0) {
      if (blk > 0) {
        syrk_tile<16>(F, ld, N, o, o, pend, o - 16, 16);
        __syncwarp();
      }
      small_leaf(F, xd, ld, o, wb, status, s, b);
    } else if (warp < blk) {
      small_xblock(F, xd, ld, o - 16, c0 + 16 * (warp - 1), pend);
    }
    if (blk > 0) {
      const int nt = trapezoid_tiles(nti, ntj);
      for (int q = take_tile(next_tile); q < nt; q = take_tile(next_tile)) {
        int i, j;
        trapezoid_tile(q, ntj, i, j);
        syrk_tile<16>(F, ld, N, o + i * TS, o + j * TS, pend, o - 16, 16);
      }
    }
    __syncthreads();
    if (tid == 0) *next_tile = nx < pend ? 1 : 0;
    if (warp == kW - 1)
      small_leaf_inverse(F, xd, ld, o, wb);
    else
      for (int r = nx + tid; r < N; r += NT - 32) small_row_solve(F, xd, ld, o, wb, r);
    __syncthreads();
  }
}
// its last row, one warp per block (those of the first warps)
template <typename T>
__device__ __forceinline__ void small_panel_last(T* F, const T* xd, int ld, int c0, int pend) {
  const int last = (pend - c0 + 15) / 16 - 1, warp = threadIdx.x >> 5;
  if (warp < last) small_xblock(F, xd, ld, c0 + 16 * last, c0 + 16 * warp, pend);
}

// Shared memory (elements) of factor_block: 64 columns and what the loops
// read past them
template <typename T>
constexpr int kBlockElems = small_ld<T>(kPanel) * kPanel + kPanel + 16;

// The diagonal block of the panel at column c0 (width w) of a front in HBM (order
// N): L is written back (lower part), D^{-1} (w x w, ld w) to inv.  sm:
// kBlockElems elements.  The blocked steps above took the place of a 64 x 64
// Cholesky with the inverse formed in three CTA-wide steps per 16 columns.
// Fronts of G = float are computed in T = double: the block is all latency, and
// the double tensor cores shorten it (in float, on the FMA units, one took
// twice as long); only its results are rounded.
template <typename T, typename G, int NT>
__device__ __noinline__ void factor_block(G* Fg, int N, int c0, int w, T* sm, G* inv, int* status,
                                          int s, int b) {
  __shared__ int next_tile;
  const int ld = small_ld<T>(kPanel);
  T* xd = sm + ld * kPanel;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kW = NT / 32;
  G* D = Fg + c0 + int64_t(c0) * N;
  if (tid == 0) next_tile = 0;
  for (int c = warp; c < w; c += kW)
    for (int r = c + lane; r < w; r += 32) sm[r + c * ld] = T(D[r + int64_t(c) * N]);
  __syncthreads();
  small_panel<T, NT>(sm, xd, ld, w, 0, w, &next_tile, status, s, b);
  small_panel_last(sm, xd, ld, 0, w);
  __syncthreads();
  for (int c = warp; c < w; c += kW)
    for (int r = lane; r < w; r += 32) {
      if (r >= c) D[r + int64_t(c) * N] = G(sm[r + c * ld]);
      inv[r + c * w] = G(xinv(sm, xd, ld, r, c));
    }
}

// T: what the front is computed in; G: what it is stored in.  Float fronts
// of up to 160 rows are computed in double, like their diagonal blocks above
// (and their entries need no rounding before the sums); larger ones in float,
// which is all that shared memory holds of them.
template <typename T, typename G, int NT>
__global__ void __launch_bounds__(NT, (sizeof(T) > 8 ? 256 : 512) / NT)
k_small_front(DevSym S, const PanelTask* __restrict__ tasks, const void* vals, int vals_dtype,
              int64_t vals_stride, G* fronts, int64_t front_stride, G* dinv,
              const int64_t* __restrict__ dinv_off, int64_t dinv_stride, int* status) {
  extern __shared__ __align__(16) unsigned char front_raw[];
  __shared__ int next_tile;
  T* F = reinterpret_cast<T*>(front_raw);
  const int s = tasks[blockIdx.x].s;
  const int b = blockIdx.y;
  const int N = S.front_n[s];
  const int ns = S.sn_first[s + 1] - S.sn_first[s];
  const int ld = small_ld<T>(N);
  T* xd = F + ld * N;
  int32_t* rel_s = reinterpret_cast<int32_t*>(xd + N + 16);   // two maps of N
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kW = NT / 32;
  const G* own = fronts + int64_t(b) * front_stride;
  G* out = fronts + int64_t(b) * front_stride + S.front_off[s];

  // Assembly.  Its cost is the latency of dependent loads, so what does not
  // depend on the predecessor (the zeros, the row maps, the children's
  // places, this thread's entries) comes before the wait, and the children's
  // values are loaded kAddCols columns at a time before they are added.
  constexpr int kEnt = 4, kAddCols = sizeof(T) > 8 ? 8 : 16;
  const int64_t a0 = S.amap_ptr[s], a1 = S.amap_ptr[s + 1];
  int pos[kEnt], ent[kEnt];
#pragma unroll
  for (int u = 0; u < kEnt; ++u) {
    const int64_t q = a0 + tid + u * NT;
    pos[u] = q < a1 ? S.amap_pos[q] : -1;
    ent[u] = q < a1 ? S.amap_e[q] : 0;
  }
  const int ch0 = S.child_ptr[s], ch1 = S.child_ptr[s + 1];
  int nbc[2] = {0, 0}, ncc[2] = {0, 0};
  const G* upd[2] = {nullptr, nullptr};
  auto meet = [&](int ci, int u) {   // child ci: its size, place and row map
    const int c = S.child[ci];
    const int nsc = S.sn_first[c + 1] - S.sn_first[c];
    ncc[u] = S.front_n[c];
    nbc[u] = ncc[u] - nsc;
    upd[u] = own + S.front_off[c] + nsc + int64_t(nsc) * ncc[u];
    const int32_t* rel = S.rel + S.rel_ptr[c];
    for (int i = tid; i < nbc[u]; i += NT) rel_s[u * N + i] = rel[i];
  };
#pragma unroll
  for (int u = 0; u < 2; ++u)
    if (ch0 + u < ch1) meet(ch0 + u, u);
  for (int i = tid; i < ld * N; i += NT) F[i] = T(0);
  __syncthreads();
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  const int64_t v0 = int64_t(b) * vals_stride;
#pragma unroll
  for (int u = 0; u < kEnt; ++u)
    if (pos[u] >= 0)
      F[pos[u] + (pos[u] / N) * (ld - N)] = load_val<T>(vals, vals_dtype, v0 + ent[u]);
  for (int64_t q = a0 + tid + kEnt * NT; q < a1; q += NT) {
    const int ps = S.amap_pos[q];
    F[ps + (ps / N) * (ld - N)] = load_val<T>(vals, vals_dtype, v0 + S.amap_e[q]);
  }
  for (int ci = ch0; ci < ch1; ci += 2) {
    if (ci > ch0) {
      __syncthreads();   // the maps are read
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (ci + u < ch1) meet(ci + u, u);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (ci + u >= ch1) break;
      __syncthreads();   // the entries and the child before
      const int nb = nbc[u], nc = ncc[u];
      const int32_t* rel = rel_s + u * N;
      for (int j0 = warp; j0 < nb; j0 += kW * kAddCols) {
        int to[kAddCols];
#pragma unroll
        for (int q = 0; q < kAddCols; ++q) to[q] = j0 + q * kW < nb ? rel[j0 + q * kW] * ld : 0;
#pragma unroll 1
        for (int i = j0 + lane; i < nb + lane; i += 32) {
          const G* src = upd[u] + min(i, nb - 1) + int64_t(j0) * nc;
          const int ri = i < nb ? rel[i] : 0;
          T v[kAddCols];
#pragma unroll
          for (int q = 0; q < kAddCols; ++q)
            v[q] = i < nb && j0 + q * kW <= i ? T(src[q * kW * nc]) : T(0);
#pragma unroll
          for (int q = 0; q < kAddCols; ++q)
            if (i < nb && j0 + q * kW <= i) F[ri + to[q]] += v[q];
        }
      }
    }
  }
  __syncthreads();

  constexpr int TS = kSyrkTile<T>;
  for (int c0 = 0; c0 < ns; c0 += kPanel) {
    const int pend = min(c0 + kPanel, ns);
    small_panel<T, NT>(F, xd, ld, N, c0, pend, &next_tile, status, s, b);
    small_panel_last(F, xd, ld, c0, pend);
    if (pend < N) {   // the rest of the front
      const int nti = (N - pend + TS - 1) / TS, nt = trapezoid_tiles(nti, nti);
      for (int q = take_tile(&next_tile); q < nt; q = take_tile(&next_tile)) {
        int i, j;
        trapezoid_tile(q, nti, i, j);
        syrk_tile<0>(F, ld, N, pend + i * TS, pend + j * TS, N, c0, pend - c0);
      }
    }
    __syncthreads();
  }
  // the lower triangle (nothing reads a front's upper part) and the panel
  // inverses, whole w x w blocks
  for (int c = warp; c < N; c += kW)
#pragma unroll 4
    for (int r = c + lane; r < N; r += 32) out[r + c * N] = G(F[r + c * ld]);
  G* inv = dinv + int64_t(b) * dinv_stride + dinv_off[s];
  for (int c = warp; c < ns; c += kW) {
    const int c0 = c / kPanel * kPanel, w = min(kPanel, ns - c0);
    G* dst = inv + int64_t(c0) * kPanel + int64_t(c - c0) * w;
    for (int r = lane; r < w; r += 32) dst[r] = G(xinv(F, xd, ld, c0 + r, c));
  }
}

}  // namespace
}  // namespace dct
