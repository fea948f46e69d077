// Fronts of general (unsymmetric-valued, structurally symmetric) float64
// plans: P A P^T = L U without row exchanges, with static pivoting -- a
// pivot whose magnitude is below floor * max|block| (floor = sqrt(eps) by
// default, the threshold of SuperLU_DIST's static pivoting) is replaced by
// that bound with the pivot's sign and counted in status[4]; a non-finite
// pivot records DCT_ERR_ZERO_PIVOT.
//
// Storage, with the layout of the symmetric plans' fronts:
//   F1 (the plan's fronts):   L's multipliers below the diagonal, 1 on it;
//   F2 (the plan's fronts2):  U^T, F2[r][c] = U[c][r] for r >= c.
// A front's boundary block (its Schur complement, the update matrix for the
// parent) keeps its lower part in F1 and its upper part, transposed, in F2,
// so extend-add, the panel TRSM and the substitution kernels of the
// symmetric plans apply to each buffer unchanged.
#pragma once
#include <cuda_runtime.h>

#include "factor_diag.cuh"
#include "front_small.cuh"

namespace dct {
namespace {

// the pivot used at step k of a general front: p itself when finite and not
// smaller than tau in magnitude, else the static replacement
__device__ __forceinline__ double static_pivot(double p, double tau, int* status, int s,
                                               int b) {
  if (!(fabs(p) < INFINITY)) {
    flag_pivot(status, s, b);
    return tau > 0.0 ? tau : 1.0;
  }
  if (fabs(p) >= tau && p != 0.0) return p;
  atomicAdd(&status[4], 1);
  const double t = tau > 0.0 ? tau : 1.0;
  return p < 0.0 ? -t : t;
}

// max over the CTA of the threads' values (NT threads, NT / 32 doubles of red)
template <int NT>
__device__ __forceinline__ double block_max(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double m = 0.0;
  for (int i = 0; i < NT / 32; ++i) m = fmax(m, red[i]);
  __syncthreads();
  return m;
}

// ---- elimination of a dense N x N block in shared memory, 16 columns at a time
// (the blocked steps of front_small.cuh for two factors): per block, one warp
// factors the 16 x 16 diagonal block, then every row below it and every column
// right of it is solved by a thread of its own, then the rest takes the
// rank-16 update on the double tensor cores.  Three barriers per 16 pivots,
// where an elimination pivot by pivot takes three per pivot.  Measured on a
// B200 (three 4,199-unknown 3-D systems): a trailing update with its diagonal
// block 39 us against 101, a level of single-CTA fronts 51 against 161.

// LU of the wb x wb block at o (wb <= 16), one warp: lane (i, h) holds the
// columns 8 h .. 8 h + 7 of row i.  rd: 1 / pivot.
__device__ __forceinline__ void lu_leaf(double* D, double* rd, int ld, int o, int wb, double tau,
                                        int* status, int s, int b) {
  const int lane = threadIdx.x & 31, i = lane & 15, h = lane >> 4;
  double v[8];
  double* row = D + (o + i) + (o + 8 * h) * ld;
  const bool in = i < wb;
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = in && 8 * h + q < wb ? row[q * ld] : 0.0;
#pragma unroll 1
  for (int k8 = 0; k8 < wb; k8 += 8)
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const int k = k8 + kk;
      if (k < wb) {
        // row k, and column k below it, as they stand
        if (i == k) {
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (8 * h + q >= k && 8 * h + q < wb) row[q * ld] = v[q];
        } else if (h == k8 / 8 && i > k && in) {
          row[kk * ld] = v[kk];
        }
        __syncwarp();
        double piv = D[(o + k) + (o + k) * ld];
        // (rows and columns beyond the block repeat its last one: they may lie
        // beyond the front, and nothing uses them)
        const double li = D[(o + min(i, wb - 1)) + (o + k) * ld];
        double u[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) u[q] = D[(o + k) + (o + min(8 * h + q, wb - 1)) * ld];
        if (!(fabs(piv) >= tau && fabs(piv) < INFINITY && piv != 0.0)) {
          if (lane == 0) piv = static_pivot(piv, tau, status, s, b);
          piv = __shfl_sync(0xffffffffu, piv, 0);
          if (lane == 0) D[(o + k) + (o + k) * ld] = piv;
        }
        const double inv = 1.0 / piv;
        if (lane == 0) rd[o + k] = inv;
        const double l = li * inv;
        __syncwarp();   // column k is read by both halves before it is replaced
        if (i > k && in) {
          if (h == 0) D[(o + i) + (o + k) * ld] = l;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (8 * h + q > k) v[q] -= l * u[q];
        }
        __syncwarp();
      }
    }
}

// D[r, c] -= sum_{16 k} D[r, k0 + k] D[k0 + k, c] on the 16 x 16 tile at (r0, c0);
// one warp
__device__ __forceinline__ void lu_tile(double* D, int ld, int N, int r0, int c0, int k0, int kw) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc[2][2][2];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 2; ++q) acc[p][q][0] = acc[p][q][1] = 0.0;
#pragma unroll
  for (int k = 0; k < 16; k += 4) {
    const bool in = k + t < kw;
    double a[2], bq[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int r = min(r0 + 8 * p + g, N - 1), c = min(c0 + 8 * p + g, N - 1);
      a[p] = in ? D[r + (k0 + k + t) * ld] : 0.0;
      bq[p] = in ? D[(k0 + k + t) + c * ld] : 0.0;
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
      for (int e = 0; e < 2; ++e) {
        const int r = r0 + 8 * p + g, c = c0 + 8 * q + 2 * t + e;
        if (r < N && c < N) D[r + c * ld] -= acc[p][q][e];
      }
}

// the first ns columns of the N x N block D eliminated: multipliers below the
// diagonal, U on and above it, the Schur complement in the rest
template <int NT>
__device__ __forceinline__ void lu_eliminate(double* D, double* rd, int ld, int N, int ns,
                                             double tau, int* status, int s, int b) {
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int o = 0; o < ns; o += 16) {
    const int wb = min(16, ns - o), nx = o + wb, nt = N - nx;
    if (warp == 0) lu_leaf(D, rd, ld, o, wb, tau, status, s, b);
    __syncthreads();
    for (int e = tid; e < 2 * nt; e += NT) {
      double v[16];
      const bool below = e < nt;
      // a row below: x U = row; a column to the right: L x = column
      double* p = below ? D + (nx + e) + o * ld : D + o + (nx + e - nt) * ld;
      const int step = below ? ld : 1;
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = q < wb ? p[q * step] : 0.0;
#pragma unroll 1
      for (int k4 = 0; k4 < wb; k4 += 4)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const int k = min(k4 + kk, wb - 1);
          // U's row or L's column beyond the pivot, registers shifted by one
          // (values shifted in from beyond the block are not used)
          const double* f = D + (o + k) + (o + k) * ld;
          const int fs = below ? ld : 1;
          const double x = below ? v[0] * rd[o + k] : v[0];
          if (k4 + kk < wb) p[k * step] = x;
#pragma unroll
          for (int j = 1; j < 16; ++j) v[j - 1] = v[j] - x * f[min(j, wb - 1 - k) * fs];
        }
    }
    __syncthreads();
    const int n16 = (nt + 15) / 16;
    for (int q = warp; q < n16 * n16; q += NT / 32)
      lu_tile(D, ld, N, nx + q % n16 * 16, nx + q / n16 * 16, o, wb);
    __syncthreads();
  }
}

// LU of the w x w diagonal block of panel p (columns c0 ..) of a general
// front (order N): D = [lower from F1 | upper from F2^T]; writes L (unit) to
// F1, U^T to F2, L^{-1} to dinv_l and (U^T)^{-1} to dinv_m (w x w, ld w).
// Needs kLuDiagElems doubles at sm.
constexpr int kLuLd = small_ld<double>(kPanel);
constexpr int kLuDiagElems = 2 * kLuLd * kPanel + 3 * kPanel + 16;
template <int NT>
__device__ __noinline__ void lu_diag(double* F1, double* F2, int N, int c0, int w, double* sm,
                                     double* dinv_l, double* dinv_m, int* status, int s, int b,
                                     double floor_rel) {
  static_assert(NT >= 256, "four warps per inverse");
  __shared__ double red[NT / 32];
  constexpr int ld = kLuLd;
  double* D = sm;                      // L and U, then L with its inverse above it
  double* M = D + ld * kPanel;         // U^T with its inverse above it
  double* rd = M + ld * kPanel;        // 1 / pivot: the inverse diagonal of U^T
  double* one = rd + kPanel;           // that of L
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kW = NT / 32;
  double mx = 0.0;
  for (int c = warp; c < w; c += kW)
    for (int r = lane; r < w; r += 32) {
      const double v = r >= c ? F1[(c0 + r) + int64_t(c0 + c) * N]
                              : F2[(c0 + c) + int64_t(c0 + r) * N];
      mx = fmax(mx, fabs(v));
      D[r + c * ld] = v;
    }
  if (tid < kPanel) one[tid] = 1.0;
  const double tau = floor_rel * block_max<NT>(mx, red);
  lu_eliminate<NT>(D, rd, ld, w, w, tau, status, s, b);
  for (int c = warp; c < w; c += kW)
    for (int r = lane; r < w; r += 32)
      if (r >= c) {
        const double u = D[c + r * ld];
        M[r + c * ld] = u;
        F1[(c0 + r) + int64_t(c0 + c) * N] = r == c ? 1.0 : D[r + c * ld];
        F2[(c0 + r) + int64_t(c0 + c) * N] = u;
      }
  __syncthreads();
  // both inverses, four warps each
  const int nblk = (w + 15) / 16, wi = warp & 3;
  double* T = warp < 4 ? D : M;
  double* td = warp < 4 ? one : rd;
  if (warp < 8 && wi < nblk) small_leaf_inverse(T, td, ld, 16 * wi, min(16, w - 16 * wi));
  for (int i = 1; i < nblk; ++i) {
    __syncthreads();
    if (warp < 8 && wi < i) small_xblock(T, td, ld, 16 * i, 16 * wi, w);
  }
  __syncthreads();
  for (int c = warp; c < w; c += kW)
    for (int r = lane; r < w; r += 32) {
      dinv_l[r + c * w] = xinv(D, one, ld, r, c);
      dinv_m[r + c * w] = xinv(M, rd, ld, r, c);
    }
}

// shared memory of a single-CTA general front: the front and the reciprocal
// pivots
__host__ __device__ constexpr size_t small_lu_smem(int N) {
  return sizeof(double) * (size_t(small_ld<double>(N)) * N + N);
}

// One CTA per general front of order N <= the single-CTA limit: assemble
// the whole front in shared memory (A's lower entries and, through the
// transpose map, its upper ones; the children's update matrices from both
// buffers), eliminate the ns pivots (the boundary block receives its Schur
// complement), and write L / U^T.
__global__ void __launch_bounds__(kThreads)
k_small_front_lu(DevSym S, const PanelTask* __restrict__ tasks, const double* vals,
                 int64_t vals_stride, const int32_t* __restrict__ tr, double* fronts,
                 double* fronts2, int64_t front_stride, int* status, double floor_rel) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[kThreads / 32];
  double* F = reinterpret_cast<double*>(smem_raw);
  const int s = tasks[blockIdx.x].s;
  const int b = blockIdx.y;
  const int N = S.front_n[s], ld = small_ld<double>(N);
  const int ns = S.sn_first[s + 1] - S.sn_first[s];
  double* rd = F + ld * N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kW = kThreads / 32;
  const int64_t off = int64_t(b) * front_stride + S.front_off[s];
  for (int i = tid; i < ld * N; i += blockDim.x) F[i] = 0.0;
  __syncthreads();
  const double* V = vals + int64_t(b) * vals_stride;
  for (int64_t q = S.amap_ptr[s] + tid; q < S.amap_ptr[s + 1]; q += blockDim.x) {
    const int pos = S.amap_pos[q];
    const int r = pos % N, c = pos / N;
    const int e = S.amap_e[q];
    F[r + c * ld] = V[e];
    if (r != c) F[c + r * ld] = V[tr[e]];
  }
  __syncthreads();
  for (int ci = S.child_ptr[s]; ci < S.child_ptr[s + 1]; ++ci) {
    const int c = S.child[ci];
    const int nc = S.front_n[c];
    const int nsc = S.sn_first[c + 1] - S.sn_first[c];
    const int nbc = nc - nsc;
    const int64_t coff = int64_t(b) * front_stride + S.front_off[c] + nsc + int64_t(nsc) * nc;
    const double* U1 = fronts + coff;
    const double* U2 = fronts2 + coff;
    const int32_t* rel = S.rel + S.rel_ptr[c];
    // a column of both update matrices per warp, four rows of each in flight
    for (int j = warp; j < nbc; j += kW) {
      const int rj = rel[j];
      for (int i0 = j + lane; i0 < nbc + lane; i0 += 128) {
        double v1[4], v2[4];
        int ri[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = i0 + 32 * q;
          ri[q] = i < nbc ? rel[i] : -1;
          v1[q] = i < nbc ? U1[i + int64_t(j) * nc] : 0.0;
          v2[q] = i < nbc && i > j ? U2[i + int64_t(j) * nc] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (ri[q] >= 0) {
            F[ri[q] + rj * ld] += v1[q];
            if (ri[q] != rj) F[rj + ri[q] * ld] += v2[q];
          }
      }
    }
    __syncthreads();
  }
  double mx = 0.0;
  for (int i = tid; i < ld * N; i += blockDim.x) mx = fmax(mx, fabs(F[i]));
  const double tau = floor_rel * block_max<kThreads>(mx, red);
  lu_eliminate<kThreads>(F, rd, ld, N, ns, tau, status, s, b);
  double* o1 = fronts + off;
  double* o2 = fronts2 + off;
  // the lower triangles (nothing reads a front's upper part)
  for (int c = warp; c < N; c += kW)
    for (int r = c + lane; r < N; r += 32) {
      o1[r + c * N] = (r == c && c < ns) ? 1.0 : F[r + c * ld];
      o2[r + c * N] = F[c + r * ld];
    }
}

}  // namespace
}  // namespace dct
