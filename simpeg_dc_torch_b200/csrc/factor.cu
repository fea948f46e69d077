// Numeric multifrontal Cholesky (A = L L^T) of nbatch systems on one pattern.
//
// Fronts are dense N x N column-major blocks (ld = N) in one buffer per
// system.  Levels of the assembly tree run bottom-up; within a level every
// front (and every system of the batch, grid.y) is independent.
//
//  * small fronts (N <= 160 f64 / 224 f32): one CTA assembles the front in
//    shared memory (zero, scatter A entries, extend-add each child's update
//    matrix in turn), runs the partial Cholesky of its ns pivot columns and
//    writes the factor panel, the update matrix and the inverses of the
//    panel's diagonal blocks (front_small.cuh);
//  * large fronts: the lower triangle is assembled from the first two
//    children in one pass, the entries are added, further children are
//    extend-added one slot per launch (so two children of a front never
//    race), then every 64-column panel is factored by a panel
//    kernel (diagonal block Cholesky + TRSM of all rows below it, one CTA per
//    64-row tile) followed by a trailing-update kernel (one CTA per 64x64
//    lower tile, C -= L_i L_j^T; in float32 plans 128x128 tensor-core tiles
//    fed from split panel images, update_tc.cu).
//
// A non-positive or NaN pivot is replaced by 1 so the factorization runs to
// the end, and the first such front is recorded in the status words; the host
// reports DCT_ERR_ZERO_PIVOT.  No device assert or trap is used.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "dct_internal.h"
#include "factor_diag.cuh"
#include "factor_lu.cuh"
#include "front_small.cuh"
#include "tile_pipe.cuh"
#include "tc_common.cuh"

namespace dct {
namespace {

// resident CTAs per SM the trailing-update kernel is compiled for: three for
// real values (two, with the output tile loaded before the products, measured
// 7 % slower), one for complex (its 4 x 4 accumulators are twice as wide)
template <typename T>
constexpr int kUpdMinBlocks = sizeof(T) > 8 ? 1 : 3;

// ------------------------------------------------------------ large: setup
// Assembly of the large fronts of a level, one warp per column of the lower
// triangle: each entry is the sum of the update matrices of the front's first
// two children at it, found through the inverse of their row maps (inv: for
// every row of the parent the child's, or -1), so that the triangle is written
// once.  Clearing it first and adding one child after the other read and wrote
// it three times (269,001-node benchmark: 1.77 against 3.29 ms in float64, 1.01
// against 1.52 in float32).  The upper triangle of a front is never read.
// task: s, p = first of kThreads / 32 columns.
template <typename T>
__global__ void __launch_bounds__(kThreads)
k_large_assemble(DevSym S, const PanelTask* __restrict__ tasks, const int32_t* __restrict__ inv,
                 const int64_t* __restrict__ inv_off, T* fronts, int64_t front_stride) {
  const int s = tasks[blockIdx.x].s;
  const int j = tasks[blockIdx.x].p + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int N = S.front_n[s];
  if (j >= N) return;
  T* base = fronts + int64_t(blockIdx.y) * front_stride;
  T* F = base + S.front_off[s] + int64_t(j) * N;
  const int ch0 = S.child_ptr[s], nch = S.child_ptr[s + 1] - ch0;
  const int32_t* map[2];
  const T* src[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    map[u] = inv + inv_off[s] + int64_t(u) * N;
    src[u] = nullptr;
    if (u < nch && map[u][j] >= 0) {
      const int c = S.child[ch0 + u];
      const int nc = S.front_n[c], nsc = S.sn_first[c + 1] - S.sn_first[c];
      src[u] = base + S.front_off[c] + nsc + int64_t(nsc + map[u][j]) * nc;
    }
  }
  constexpr int kBatch = 8;   // rows of a lane in flight
  for (int i0 = j + lane; i0 < N; i0 += kBatch * 32) {
    T v[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q) {
      const int i = i0 + 32 * q;
      int at[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) at[u] = i < N && src[u] != nullptr ? map[u][i] : -1;
      v[q] = at[0] >= 0 ? src[0][at[0]] : T(0);
      if (at[1] >= 0) v[q] += src[1][at[1]];
    }
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (i0 + 32 * q < N) F[i0 + 32 * q] = v[q];
  }
}

// The matrix entries, added to what the children left; general plans (fronts2
// non-null): the transposed entries, through the transpose map tr, go to the
// same positions of fronts2 (U^T's buffer)
template <typename T>
__global__ void __launch_bounds__(kThreads)
k_large_scatter(DevSym S, const PanelTask* __restrict__ tasks, const void* vals,
                int vals_dtype, int64_t vals_stride, T* fronts,
                int64_t front_stride, T* fronts2, const int32_t* __restrict__ tr) {
  const int s = tasks[blockIdx.x].s;
  const int b = blockIdx.y;
  T* F = fronts + int64_t(b) * front_stride + S.front_off[s];
  T* F2 = fronts2 == nullptr ? nullptr : fronts2 + int64_t(b) * front_stride + S.front_off[s];
  const int64_t a0 = S.amap_ptr[s], a1 = S.amap_ptr[s + 1];
  for (int64_t q = a0 + blockIdx.z * kThreads + threadIdx.x; q < a1; q += gridDim.z * kThreads) {
    F[S.amap_pos[q]] += load_val<T>(vals, vals_dtype, int64_t(b) * vals_stride + S.amap_e[q]);
    if (F2 != nullptr)
      F2[S.amap_pos[q]] += load_val<T>(vals, vals_dtype,
                                       int64_t(b) * vals_stride + tr[S.amap_e[q]]);
  }
}

// The update matrices of children beyond the second, one child slot per launch.
// task: s = parent, t0 = child, t1 = first column of the child's update
// matrix handled by this CTA (8 columns, one warp each)
template <typename T>
__global__ void __launch_bounds__(kThreads)
k_large_extend_add(DevSym S, const PanelTask* __restrict__ tasks, T* fronts,
                   int64_t front_stride) {
  const PanelTask tk = tasks[blockIdx.x];
  const int b = blockIdx.y;
  const int s = tk.s, c = tk.t0;
  const int N = S.front_n[s];
  const int nc = S.front_n[c];
  const int nsc = S.sn_first[c + 1] - S.sn_first[c];
  const int nbc = nc - nsc;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = tk.t1 + warp;
  if (j >= nbc) return;
  T* F = fronts + int64_t(b) * front_stride + S.front_off[s];
  const T* U = fronts + int64_t(b) * front_stride + S.front_off[c];
  const int32_t* rel = S.rel + S.rel_ptr[c];
  const int64_t dst_col = int64_t(rel[j]) * N;
  const T* src = U + (nsc + j) * int64_t(nc) + nsc;
  for (int i = j + lane; i < nbc; i += 32) F[rel[i] + dst_col] += src[i];
}

// ------------------------------------------------------------ large: panels
constexpr int kPanelLd = kPanel + 4;   // 4 modulo 8: see dmma.cuh
// task: s, p, t0 >= 1: the 64-row tile t0-1 below panel p becomes
// F_rows D_p^{-T}, using the inverse stored when the diagonal was factored.
// Float32 plans (im.img non-null) also write the rows' split image
// (hi = tf32(x), lo = x - hi) for the tensor-core trailing update; the
// image's padding rows and the columns beyond a narrow panel stay zero from
// the plan's creation.
template <typename T>
__global__ void __launch_bounds__(kThreads)
k_large_panel(DevSym S, const PanelTask* __restrict__ tasks, T* fronts,
              int64_t front_stride, const T* dinv, const int64_t* dinv_off,
              int64_t dinv_stride, ImgArgs im) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* S1 = reinterpret_cast<T*>(smem_raw);   // [q][c] = Dinv[c, q]
  T* S2 = S1 + kPanel * kPanelLd;           // [q][r] = F[r, q]
  const PanelTask tk = tasks[blockIdx.x];
  const int b = blockIdx.y;
  const int s = tk.s;
  const int N = S.front_n[s];
  const int ns = S.sn_first[s + 1] - S.sn_first[s];
  const int c0 = tk.p * kPanel;
  const int w = min(kPanel, ns - c0);
  T* F = fronts + int64_t(b) * front_stride + S.front_off[s];
  const T* Di = dinv + int64_t(b) * dinv_stride + dinv_off[s] +
                int64_t(tk.p) * kPanel * kPanel;
  const int r0 = c0 + w + (tk.t0 - 1) * kPanel;
  const int nr = min(kPanel, N - r0);
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  small_load_cols(S1, kPanelLd, Di, w, w, w);
  small_load_cols(S2, kPanelLd, F + r0 + int64_t(c0) * N, N, nr, w);
  small_commit();
  small_wait<0>();
  __syncthreads();
  // float: neighbours store neighbouring rows of F and of the images (with runs
  // of rows per thread the panels of the 269,001-node benchmark took 3.9 ms for 2.5)
  std::conditional_t<sizeof(T) == 4, StridedTile<T, kPanel>, SmallTile<T, kPanel>> acc;
  acc.zero();
  acc.template mul<false>(S1, kPanelLd, S2, (w + 3) & ~3, w, nr);
  float* img = nullptr;
  int R0 = 0, G = 0;
  if constexpr (sizeof(T) == 4) {
    if (im.img != nullptr) {
      img = im.img + int64_t(b) * im.stride + im.off[im.pan_first[s] + tk.p];
      R0 = img_origin(tk.p, ns);
      G = img_groups(tk.p, ns, N);
    }
  }
  acc.each(w, [&](int c, int r, T& x) {
    if (c >= w || r >= nr) return;
    F[(r0 + r) + int64_t(c0 + c) * N] = x;
    if constexpr (sizeof(T) == 4) {
      if (img == nullptr) return;
      const int gr = r0 + r - R0;
      const float v = float(x);
      const uint32_t h = tf32_rna(v);
      img[img_index(G, 0, c / kImgK, gr >> 3, c % kImgK, gr & 7)] = __uint_as_float(h);
      img[img_index(G, 1, c / kImgK, gr >> 3, c % kImgK, gr & 7)] = v - __uint_as_float(h);
    }
  });
}

// task: s, p, t0 = i, t1 = j (i >= j): 64 x 64 tile of the trailing block
// that starts after panel p, F_ij -= L_i L_j^T over the columns of
// update_range.
// The CTA of tile (0, 0) -- the next panel's diagonal block -- factors that
// block after its own update (no other task of the launch touches it).
// t0 = -1: factor the diagonal block of panel p itself (a front's first panel).
constexpr int kUT = kUpdateTile;

// One tile update F_out[i, j] -= Fa_i Fb_j^T over the columns ka .. base - 1:
// rows rj.. of Fb and ri.. of Fa, entries on or below the diagonal.
template <typename T>
__device__ __forceinline__ void tile_update(const T* Fa, const T* Fb, T* Fo, int N, int ka,
                                            int base, int ri, int rj, int ni, int nj, T* ring) {
  SmallTile<T, kUT> cur, acc;
  acc.zero();
  ColStream<T, kUT> a(Fb + rj + int64_t(ka) * N, N, nj), b(Fa + ri + int64_t(ka) * N, N, ni);
  TilePipe<T, kUT, false>::run(ring, base - ka, nj, ni, acc, a, b);
  cur.each(nj, [&](int c, int r, T& v) {
    v = c < nj && r < ni && ri + r >= rj + c ? Fo[(ri + r) + int64_t(rj + c) * N] : T(0);
  });
  tile_subtract(cur, acc);
  cur.each(nj, [&](int c, int r, T& v) {
    if (c < nj && r < ni && ri + r >= rj + c) Fo[(ri + r) + int64_t(rj + c) * N] = v;
  });
}

// General plans (fronts2 non-null, float64): two products per tile, the lower
// part of the trailing block in F1 -= L_i U_j^T-rows and its upper part,
// transposed in F2, -= U^T_i L_j^T; diagonal blocks by lu_diag.
template <typename T>
__global__ void __launch_bounds__(kThreads, kUpdMinBlocks<T>)
k_large_update(DevSym S, const PanelTask* __restrict__ tasks, T* fronts,
               int64_t front_stride, T* dinv, const int64_t* dinv_off,
               int64_t dinv_stride, int bpan, int* status, T* fronts2, T* dinv2,
               double pivot_floor) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  const PanelTask tk = tasks[blockIdx.x];
  const int b = blockIdx.y;
  const int s = tk.s;
  const int N = S.front_n[s];
  const int ns = S.sn_first[s + 1] - S.sn_first[s];
  const int c0 = tk.p * kPanel;
  const int w = min(kPanel, ns - c0);
  const int base = c0 + w;
  T* F = fronts + int64_t(b) * front_stride + S.front_off[s];
  T* Dv = dinv + int64_t(b) * dinv_stride + dinv_off[s];
  T* F2 = nullptr;
  T* Dv2 = nullptr;
  if constexpr (sizeof(T) == 8) {
    if (fronts2 != nullptr) {
      F2 = fronts2 + int64_t(b) * front_stride + S.front_off[s];
      Dv2 = dinv2 + int64_t(b) * dinv_stride + dinv_off[s];
    }
  }
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  // the diagonal block of panel q (Cholesky and inverse, or LU and both
  // inverses)
  auto diag = [&](int q) {
    const int cq = q * kPanel, wq = min(kPanel, ns - cq);
    if constexpr (sizeof(T) == 8) {
      if (F2 != nullptr) {
        lu_diag<kThreads>(reinterpret_cast<double*>(F), reinterpret_cast<double*>(F2), N, cq,
                          wq, reinterpret_cast<double*>(ring),
                          reinterpret_cast<double*>(Dv + int64_t(q) * kPanel * kPanel),
                          reinterpret_cast<double*>(Dv2 + int64_t(q) * kPanel * kPanel),
                          status, s, b, pivot_floor);
        return;
      }
    }
    factor_block<T, T, kThreads>(F, N, cq, wq, ring, Dv + int64_t(q) * kPanel * kPanel, status, s,
                              b);
  };
  if (tk.t0 < 0) {
    diag(tk.p);
    return;
  }
  const UpdateRange R = update_range(tk.p, ns, N, bpan);
  const int ri = base + tk.t0 * kUT, rj = base + tk.t1 * kUT;
  const int ni = min(kUT, N - ri), nj = min(kUT, R.cend - rj);
  if (F2 == nullptr) {
    tile_update<T>(F, F, F, N, R.ka, base, ri, rj, ni, nj, ring);
  } else {
    tile_update<T>(F, F2, F, N, R.ka, base, ri, rj, ni, nj, ring);
    tile_update<T>(F2, F, F2, N, R.ka, base, ri, rj, ni, nj, ring);
  }
  if (tk.t0 == 0 && tk.t1 == 0 && base < ns) {
    __syncthreads();   // this CTA's updates of the block are complete
    diag(tk.p + 1);
  }
}

// task: s, p.  The inverse of the factored diagonal block of panel p of a small
// general front (L, or U^T with its diagonal), written column-major (ld w) at
// dinv + dinv_off[s] + p*64*64, by the steps of front_small.cuh.
__global__ void __launch_bounds__(kThreads)
k_panel_inverse(DevSym S, const PanelTask* __restrict__ tasks, const double* fronts,
                int64_t front_stride, double* dinv, const int64_t* dinv_off,
                int64_t dinv_stride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* L = reinterpret_cast<double*>(smem_raw);
  constexpr int ld = small_ld<double>(kPanel), kW = kThreads / 32;
  double* xd = L + ld * kPanel;
  const PanelTask tk = tasks[blockIdx.x];
  const int b = blockIdx.y;
  const int s = tk.s;
  const int N = S.front_n[s];
  const int ns = S.sn_first[s + 1] - S.sn_first[s];
  const int c0 = tk.p * kPanel;
  const int w = min(kPanel, ns - c0), nblk = (w + 15) / 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* F = fronts + int64_t(b) * front_stride + S.front_off[s] + c0 + int64_t(c0) * N;
  for (int c = warp; c < w; c += kW)
    for (int r = c + lane; r < w; r += 32) {
      const double v = F[r + int64_t(c) * N];
      L[r + c * ld] = v;
      if (r == c) xd[c] = 1.0 / v;
    }
  __syncthreads();
  if (warp < nblk) small_leaf_inverse(L, xd, ld, 16 * warp, min(16, w - 16 * warp));
  for (int i = 1; i < nblk; ++i) {
    __syncthreads();
    if (warp < i) small_xblock(L, xd, ld, 16 * i, 16 * warp, w);
  }
  __syncthreads();
  double* out = dinv + int64_t(b) * dinv_stride + dinv_off[s] + int64_t(tk.p) * kPanel * kPanel;
  for (int c = warp; c < w; c += kW)
    for (int r = lane; r < w; r += 32) out[r + c * w] = xinv(L, xd, ld, r, c);
}

// ------------------------------------------------------------ supernode inverses
// L_ss^{-1} (ns x ns, column-major, ld ns) of every supernode wider than one
// panel, by recursive doubling from the panel inverses (see the schedule in
// capi.cu).  Blocks of 64 x 64 tiles; K loops skip the zero upper blocks.  Both
// products are computed transposed, (column, row), so that the lanes of a
// store run along the rows.
struct LinvArgs {
  DevSym S;
  const PanelTask* tasks;
  int64_t front_stride;
  const int64_t* dinv_off;
  int64_t dinv_stride;
  const int64_t* linv_off;
  int64_t linv_stride;
  int h;
};

template <typename T>
__global__ void __launch_bounds__(kThreads)
k_linv_init(LinvArgs g, const T* dinv, T* linv) {
  const PanelTask tk = g.tasks[blockIdx.x];
  const int b = blockIdx.y;
  const int s = tk.s;
  const int ns = g.S.sn_first[s + 1] - g.S.sn_first[s];
  const int c0 = tk.p * kPanel, w = min(kPanel, ns - c0);
  const T* Di = dinv + int64_t(b) * g.dinv_stride + g.dinv_off[s] + int64_t(tk.p) * kPanel * kPanel;
  T* X = linv + int64_t(b) * g.linv_stride + g.linv_off[s];
  for (int idx = threadIdx.x; idx < w * w; idx += blockDim.x) {
    const int r = idx % w, c = idx / w;
    X[(c0 + r) + int64_t(c0 + c) * ns] = Di[r + c * w];
  }
}

// T[d-block, a-block] = C A^{-1}: C = L[d0.., a0..] (front rows), A^{-1} the
// top block's inverse.  out tile (rt, ct): rows d0 + 64 rt, cols a0 + 64 ct.
template <typename T>
__global__ void __launch_bounds__(kThreads, kUpdMinBlocks<T>)
k_linv_t(LinvArgs g, const T* fronts, const T* linv, T* ltmp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PanelTask tk = g.tasks[blockIdx.x];
  const int b = blockIdx.y;
  const int s = tk.s, h = g.h;
  const DevSym& S = g.S;
  const int N = S.front_n[s];
  const int ns = S.sn_first[s + 1] - S.sn_first[s];
  const int a0 = 2 * tk.p * h, d0 = a0 + h;
  const int hd = min(h, ns - d0);
  const int r0 = tk.t0 * kPanel, cc0 = tk.t1 * kPanel;
  const int nr = min(kPanel, hd - r0);
  const T* F = fronts + int64_t(b) * g.front_stride + S.front_off[s];
  const T* X = linv + int64_t(b) * g.linv_stride + g.linv_off[s];
  T* Tt = ltmp + int64_t(b) * g.linv_stride + g.linv_off[s];
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  SmallTile<T, kPanel> acc;   // (column, row) of the tile
  acc.zero();
  // column c of A^{-1} starts at row c: K from the tile's first column on
  RowStream<T> inv(X + (a0 + cc0) + int64_t(a0 + cc0) * ns, ns, kPanel);
  ColStream<T, kPanel> c(F + (d0 + r0) + int64_t(a0 + cc0) * N, N, nr);
  TilePipe<T, kPanel, true>::run(reinterpret_cast<T*>(smem_raw), h - cc0, kPanel, nr, acc, inv, c);
  acc.each(kPanel, [&](int col, int r, T& v) {
    if (r < nr) Tt[(d0 + r0 + r) + int64_t(a0 + cc0 + col) * ns] = v;
  });
}

// X[d-block, a-block] = -D^{-1} T with D^{-1} the bottom block's inverse.
template <typename T>
__global__ void __launch_bounds__(kThreads, kUpdMinBlocks<T>)
k_linv_x(LinvArgs g, const T* ltmp, T* linv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PanelTask tk = g.tasks[blockIdx.x];
  const int b = blockIdx.y;
  const int s = tk.s, h = g.h;
  const int ns = g.S.sn_first[s + 1] - g.S.sn_first[s];
  const int a0 = 2 * tk.p * h, d0 = a0 + h;
  const int hd = min(h, ns - d0);
  const int r0 = tk.t0 * kPanel, cc0 = tk.t1 * kPanel;
  const int nr = min(kPanel, hd - r0);
  T* X = linv + int64_t(b) * g.linv_stride + g.linv_off[s];
  const T* Tt = ltmp + int64_t(b) * g.linv_stride + g.linv_off[s];
  pdl_wait();
  pdl_trigger();
  SmallTile<T, kPanel> acc;
  acc.zero();
  RowStream<T> t(Tt + d0 + int64_t(a0 + cc0) * ns, ns, kPanel);
  ColStream<T, kPanel> d(X + (d0 + r0) + int64_t(d0) * ns, ns, nr);
  TilePipe<T, kPanel, true>::run(reinterpret_cast<T*>(smem_raw), min(hd, r0 + kPanel), kPanel, nr,
                                 acc, t, d);
  acc.each(kPanel, [&](int col, int r, T& v) {
    if (r < nr) X[(d0 + r0 + r) + int64_t(a0 + cc0 + col) * ns] = -v;
  });
}

template <typename T>
cudaError_t run_linv(dct_plan* P, cudaStream_t st, const void* fronts, const void* dinv,
                     void* linv) {
  const int nb = P->nbatch;
  const size_t smem = sizeof(T) * TilePipe<T, kPanel, true>::kElems;
  cudaError_t e = allow_smem(P, k_linv_t<T>);
  if (e == cudaSuccess) e = allow_smem(P, k_linv_x<T>);
  if (e != cudaSuccess) return e;
  LinvArgs g{P->ds, nullptr, P->front_stride, P->d_dinv_off, P->dinv_stride,
             P->d_linv_off, P->linv_stride, 0};
  for (size_t li = 0; li < P->linv_sched.launches.size(); ++li) {
    const Launch& L = P->linv_sched.launches[li];
    if (L.count <= 0) continue;
    if ((e = P->prof.begin(L.kind, 0.0, 0.0, st)) != cudaSuccess) return e;
    g.tasks = P->linv_sched.d_tasks + L.first;
    g.h = L.arg;
    dim3 grid(static_cast<unsigned>(L.count), nb);
    if (L.kind == kLinvInit)
      k_linv_init<T><<<grid, kThreads, 0, st>>>(g, static_cast<const T*>(dinv),
                                               static_cast<T*>(linv));
    else if (L.kind == kLinvT)
      e = launch_pdl(k_linv_t<T>, grid, dim3(kThreads), smem, st, g, static_cast<const T*>(fronts),
                     static_cast<const T*>(linv), static_cast<T*>(P->ltmp));
    else
      e = launch_pdl(k_linv_x<T>, grid, dim3(kThreads), smem, st, g,
                     static_cast<const T*>(P->ltmp), static_cast<T*>(linv));
    if (e != cudaSuccess) return e;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = P->prof.end(st)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// one launch of single-CTA fronts of order up to n
template <typename T, typename G>
struct SmallLaunch {
  dct_plan* P;
  const PanelTask* tasks;
  const void* vals;
  int vals_dtype;
  int64_t vals_stride;
  dim3 grid;
  cudaStream_t st;
  cudaError_t operator()(int n) const {
    const bool narrow = n <= kSmallNarrow;
    auto fn = narrow ? k_small_front<T, G, kThreads / 2> : k_small_front<T, G, kThreads>;
    const cudaError_t e = allow_smem(P, fn);
    if (e != cudaSuccess) return e;
    return launch_pdl(fn, grid, dim3(narrow ? kThreads / 2 : kThreads), small_smem<T>(n), st, P->ds,
                      tasks, vals, vals_dtype, vals_stride, static_cast<G*>(P->fronts),
                      P->front_stride, static_cast<G*>(P->dinv),
                      static_cast<const int64_t*>(P->d_dinv_off), P->dinv_stride, P->status);
  }
};

template <typename T>
cudaError_t factor_impl(dct_plan* P, const void* vals, int vals_dtype,
                        int64_t vals_stride, cudaStream_t st) {
  T* fronts = static_cast<T*>(P->fronts);
  // general plans (float64 only): U^T's buffer
  const bool lu = sizeof(T) == 8 && P->lu != 0;
  T* fronts2 = lu ? static_cast<T*>(P->fronts2) : nullptr;
  const int nb = P->nbatch;
  cudaError_t e = cudaSuccess;
  const size_t panel_smem = sizeof(T) * (2 * kPanel * kPanelLd);
  // the update kernel's copy ring, or the diagonal block's workspace
  const size_t update_smem =
      sizeof(T) * std::max(TilePipe<T, kUT, false>::kElems, lu ? kLuDiagElems : kBlockElems<T>);
  if constexpr (sizeof(T) == 8) {
    if (lu) e = allow_smem(P, k_small_front_lu);
  }
  if (e == cudaSuccess) e = allow_smem(P, k_large_panel<T>);
  if constexpr (sizeof(T) != 4) {
    if (e == cudaSuccess) e = allow_smem(P, k_large_update<T>);
  }
  if (e != cudaSuccess) return e;
  const PanelTask* tasks = P->fact.d_tasks;
  for (size_t li = 0; li < P->fact.launches.size(); ++li) {
    const Launch& L = P->fact.launches[li];
    if (L.count <= 0) continue;
    e = P->prof.begin(L.kind, P->fact.flops[li] * nb, P->fact.bytes[li] * nb, st);
    if (e != cudaSuccess) return e;
    // grid.x is limited to 2^31-1, far above any task count here
    dim3 grid(static_cast<unsigned>(L.count), nb);
    const PanelTask* t = tasks + L.first;
    switch (L.kind) {
      case kSmallFront: {
        if constexpr (sizeof(T) == 8) {
          if (lu) {
            k_small_front_lu<<<grid, kThreads, small_lu_smem(L.arg), st>>>(
                P->ds, t, static_cast<const double*>(vals), vals_stride, P->d_tr,
                reinterpret_cast<double*>(fronts), reinterpret_cast<double*>(fronts2),
                P->front_stride, P->status, P->pivot_floor);
            break;
          }
        }
        SmallLaunch<T, T> go{P, t, vals, vals_dtype, vals_stride, grid, st};
        if constexpr (sizeof(T) == 4)
          e = L.arg <= kSmallFrontF64
                  ? SmallLaunch<double, T>{P, t, vals, vals_dtype, vals_stride, grid, st}(L.arg)
                  : go(L.arg);
        else
          e = go(L.arg);
        if (e != cudaSuccess) return e;
        break;
      }
      case kLargeScatter:
        for (T* buf : {fronts, fronts2}) {
          if (buf == nullptr) continue;
          k_large_assemble<T><<<dim3(static_cast<unsigned>(P->asm_count[li]), nb), kThreads, 0,
                                st>>>(P->ds, P->d_asm + P->asm_first[li], P->d_inv, P->d_inv_off,
                                      buf, P->front_stride);
        }
        k_large_scatter<T><<<dim3(grid.x, grid.y, 8), kThreads, 0, st>>>(
            P->ds, t, vals, vals_dtype, vals_stride, fronts, P->front_stride, fronts2,
            P->d_tr);
        break;
      case kLargeExtendAdd:
        for (T* buf : {fronts, fronts2}) {
          if (buf == nullptr) continue;
          k_large_extend_add<T><<<grid, kThreads, 0, st>>>(P->ds, t, buf, P->front_stride);
        }
        break;
      case kLargePanel:
        // general plans: L's rows take (U^T)^{-1} (L21 = A21 U11^{-1}), U^T's
        // rows take L^{-1} (U12^T = A12^T L11^{-T})
        e = launch_pdl(k_large_panel<T>, grid, dim3(kThreads), panel_smem, st, P->ds, t, fronts,
                       P->front_stride, static_cast<const T*>(lu ? P->dinv2 : P->dinv),
                       P->d_dinv_off, P->dinv_stride, sizeof(T) == 4 ? P->img : ImgArgs{});
        if (e == cudaSuccess && lu)
          e = launch_pdl(k_large_panel<T>, grid, dim3(kThreads), panel_smem, st, P->ds, t,
                         fronts2, P->front_stride, static_cast<const T*>(P->dinv),
                         P->d_dinv_off, P->dinv_stride, ImgArgs{});
        if (e != cudaSuccess) return e;
        break;
      case kLargeUpdate:
        if constexpr (sizeof(T) == 4) {
          e = launch_update_tc(
              P, t, L.count, li < P->update_nspec.size() ? P->update_nspec[li] : -1, st);
        } else {
          e = launch_pdl(k_large_update<T>, grid, dim3(kThreads), update_smem, st, P->ds, t,
                         fronts, P->front_stride, static_cast<T*>(P->dinv), P->d_dinv_off,
                         P->dinv_stride, P->update_bpan, P->status, fronts2,
                         static_cast<T*>(P->dinv2), P->pivot_floor);
        }
        if (e != cudaSuccess) return e;
        break;
      default:
        return cudaErrorInvalidValue;
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = P->prof.end(st);
    if (e != cudaSuccess) return e;
  }
  // general plans: inverses of the diagonal blocks of small fronts, for the
  // substitution (the symmetric types' fronts, and large ones, store theirs
  // while factoring)
  if constexpr (sizeof(T) == 8) {
    const int64_t ninv = int64_t(P->inv.tasks.size());
    if (lu && ninv > 0) {
      const size_t inv_smem = sizeof(T) * kBlockElems<T>;
      e = allow_smem(P, k_panel_inverse);
      if (e == cudaSuccess) e = P->prof.begin(kPanelInverse, 0.0, 0.0, st);
      if (e != cudaSuccess) return e;
      const dim3 grid(static_cast<unsigned>(ninv), nb);
      k_panel_inverse<<<grid, kThreads, inv_smem, st>>>(
          P->ds, P->inv.d_tasks, fronts, P->front_stride, static_cast<double*>(P->dinv),
          P->d_dinv_off, P->dinv_stride);
      k_panel_inverse<<<grid, kThreads, inv_smem, st>>>(
          P->ds, P->inv.d_tasks, fronts2, P->front_stride, static_cast<double*>(P->dinv2),
          P->d_dinv_off, P->dinv_stride);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = P->prof.end(st);
      if (e != cudaSuccess) return e;
    }
  }
  e = run_linv<T>(P, st, P->fronts, P->dinv, P->linv);
  if (e == cudaSuccess && lu) e = run_linv<T>(P, st, P->fronts2, P->dinv2, P->linv2);
  return e;
}

}  // namespace

cudaError_t run_factor(dct_plan* P, const void* vals, int vals_dtype,
                       int64_t vals_stride, cudaStream_t st) {
  if (P->dtype == DCT_F64)
    return factor_impl<double>(P, vals, vals_dtype, vals_stride, st);
  if (P->dtype == DCT_C128)
    return factor_impl<cplx>(P, vals, vals_dtype, vals_stride, st);
  return factor_impl<float>(P, vals, vals_dtype, vals_stride, st);
}

}  // namespace dct
