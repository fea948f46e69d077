// Multi-RHS supernodal substitution L L^T x = b for nbatch systems, in the
// permuted order, on row-major (n, k) right-hand sides.
//
// Per tree level (forward bottom-up, backward top-down):
//   supernodes of one panel (ns <= 64): one CTA per supernode, system and one
//     or more chunks of up to 64 right-hand sides does the whole step with the
//     stored panel inverse D^{-1} (solve_small.cuh);
//   larger supernodes: products with the explicit supernode inverse
//     L_ss^{-1} (formed after the factorization) and with the boundary block
//     L_Bs, in 64-row tiles (float64 on the double tensor cores, complex on the
//     FMA units: k_fwd_linv, k_fwd_bnd, k_bwd_gemm, k_bwd_linv) or in 128-row
//     tiles (float32 plans, solve_tc.cu).
//
// Two work buffers A and B of nbatch*n*k elements are used so that no launch
// ever reads a location that another CTA of the same launch writes:
//   forward:  b lives in A and receives the updates -L_Bs y_s of the rows
//             below (atomics: several supernodes of a level may share
//             ancestor rows); y_s goes to B.
//   backward: y_s -= L_Bs^T x_B with x_B (rows of ancestors, final) in A;
//             x_s = L_ss^{-T} y_s goes to A.
// The tensor-core kinds split long K ranges over CTAs and accumulate with
// atomics, so in float32 plans the rows of the supernodes that take them are
// cleared in B before the forward pass and in A (whose right-hand side is
// consumed by then) before the backward pass.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "dct_internal.h"
#include "solve_small.cuh"
#include "tile_pipe.cuh"

namespace dct {
namespace {

// ------------------------------------------------------------ large supernodes
// 64 rows of output x NC right-hand sides per CTA, K through the copy ring of
// tile_pipe.cuh (float64 and complex plans; float32: solve_tc.cu).  V elements
// of the right-hand sides are copied at a time: 16 bytes where their rows are
// aligned, else one.
template <typename T>
constexpr int kLargeCtas = sizeof(T) == 8 ? 3 : 1;

// y_s = L_ss^{-1} b_s, rows 64 t0 .. (B <- A rows)
template <typename T, int NC, int V>
__global__ void __launch_bounds__(kThreads, kLargeCtas<T>) k_fwd_linv(SolveArgs<T> g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PanelTask tk = g.tasks[blockIdx.x / g.nchunk];
  const int b = blockIdx.y;
  const int j0 = (blockIdx.x % g.nchunk) * NC;
  const int rc = min(NC, g.k - j0);
  const DevSym& S = g.S;
  const int s = tk.s;
  const int first = S.sn_first[s];
  const int ns = S.sn_first[s + 1] - first;
  const int r0 = tk.t0 * kPanel, nr = min(kPanel, ns - r0);
  const T* X = g.linv + int64_t(b) * g.linv_stride + g.linv_off[s];
  const T* A = g.A + int64_t(b) * g.n * g.k;
  T* Bo = g.B + int64_t(b) * g.n * g.k;
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  SmallTile<T, NC> acc;
  acc.zero();
  if (!rhs_reaches(g, s, b)) {   // y = 0
    acc.each(nr, [&](int r, int j, T& v) {
      if (r < nr && j < rc) Bo[int64_t(first + r0 + r) * g.k + j0 + j] = v;
    });
    return;
  }
  ColStream<T, kPanel> a(X + r0, ns, nr);
  RhsStream<T, NC, V, false> x(A, g.k, j0, rc, first, nullptr);
  TilePipe<T, NC, false>::run(reinterpret_cast<T*>(smem_raw), r0 + nr, nr, rc, acc, a, x);
  acc.each(nr, [&](int r, int j, T& v) {
    if (r < nr && j < rc) Bo[int64_t(first + r0 + r) * g.k + j0 + j] = v;
  });
}

// x_s = L_ss^{-T} y_s, rows 64 t0 .. (A <- B rows)
template <typename T, int NC, int V>
__global__ void __launch_bounds__(kThreads, kLargeCtas<T>) k_bwd_linv(SolveArgs<T> g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PanelTask tk = g.tasks[blockIdx.x / g.nchunk];
  const int b = blockIdx.y;
  const int j0 = (blockIdx.x % g.nchunk) * NC;
  const int rc = min(NC, g.k - j0);
  const DevSym& S = g.S;
  const int s = tk.s;
  const int first = S.sn_first[s];
  const int ns = S.sn_first[s + 1] - first;
  const int r0 = tk.t0 * kPanel, nr = min(kPanel, ns - r0);
  const T* X = g.linv + int64_t(b) * g.linv_stride + g.linv_off[s];
  T* A = g.A + int64_t(b) * g.n * g.k;
  const T* Bo = g.B + int64_t(b) * g.n * g.k;
  pdl_wait();
  pdl_trigger();
  SmallTile<T, NC> acc;
  acc.zero();
  RowStream<T> a(X + r0 + int64_t(r0) * ns, ns, nr);
  RhsStream<T, NC, V, false> x(Bo, g.k, j0, rc, first + r0, nullptr);
  TilePipe<T, NC, true>::run(reinterpret_cast<T*>(smem_raw), ns - r0, nr, rc, acc, a, x);
  acc.each(nr, [&](int r, int j, T& v) {
    if (r < nr && j < rc) A[int64_t(first + r0 + r) * g.k + j0 + j] = v;
  });
}

// the boundary rows ns + 64 t0 .. (in A) receive -L[rows, 0:ns] y_s, one atomic
// update per element
template <typename T, int NC, int V>
__global__ void __launch_bounds__(kThreads, kLargeCtas<T>) k_fwd_bnd(SolveArgs<T> g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PanelTask tk = g.tasks[blockIdx.x / g.nchunk];
  const int b = blockIdx.y;
  const int j0 = (blockIdx.x % g.nchunk) * NC;
  const int rc = min(NC, g.k - j0);
  const DevSym& S = g.S;
  const int s = tk.s;
  const int N = S.front_n[s], first = S.sn_first[s];
  const int ns = S.sn_first[s + 1] - first;
  const int r0 = ns + tk.t0 * kPanel, nr = min(kPanel, N - r0);
  const T* F = g.fronts + int64_t(b) * g.front_stride + S.front_off[s];
  const int32_t* rows = S.rows + S.rows_ptr[s] + r0;
  T* A = g.A + int64_t(b) * g.n * g.k;
  const T* Bo = g.B + int64_t(b) * g.n * g.k;
  pdl_wait();
  pdl_trigger();
  if (!rhs_reaches(g, s, b)) return;
  SmallTile<T, NC> acc;
  acc.zero();
  ColStream<T, kPanel> a(F + r0, N, nr);
  RhsStream<T, NC, V, false> x(Bo, g.k, j0, rc, first, nullptr);
  TilePipe<T, NC, false>::run(reinterpret_cast<T*>(smem_raw), ns, nr, rc, acc, a, x);
  acc.each(nr, [&](int r, int j, T& v) {
    if (r < nr && j < rc) atomicAdd(A + int64_t(rows[r]) * g.k + j0 + j, -v);
  });
}

// y_p (B) -= L[boundary rows, panel p]^T x[boundary rows]; a row list of at most
// nrows rows (kGemmRows, or the launch's longest) is kept in shared memory
constexpr int kGemmRows = 6144;
template <typename T, int NC, int V>
__global__ void __launch_bounds__(kThreads, kLargeCtas<T>)
k_bwd_gemm(SolveArgs<T> g, int nrows) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  int32_t* rows_s = reinterpret_cast<int32_t*>(ring + TilePipe<T, NC, true>::kElems);
  const PanelTask tk = g.tasks[blockIdx.x / g.nchunk];
  const int b = blockIdx.y;
  const int j0 = (blockIdx.x % g.nchunk) * NC;
  const int rc = min(NC, g.k - j0);
  const DevSym& S = g.S;
  const int s = tk.s;
  const int N = S.front_n[s], first = S.sn_first[s];
  const int ns = S.sn_first[s + 1] - first;
  const int c0 = tk.p * kPanel, w = min(kPanel, ns - c0);
  const T* F = g.fronts + int64_t(b) * g.front_stride + S.front_off[s];
  const int32_t* rows = S.rows + S.rows_ptr[s] + ns;
  const T* A = g.A + int64_t(b) * g.n * g.k;
  T* Bo = g.B + int64_t(b) * g.n * g.k;
  if (N - ns <= nrows)
    for (int i = threadIdx.x; i < N - ns; i += kThreads) rows_s[i] = rows[i];
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  SmallTile<T, NC> y, acc;
  y.each(w, [&](int c, int j, T& v) {
    v = c < w && j < rc ? Bo[int64_t(first + c0 + c) * g.k + j0 + j] : T(0);
  });
  acc.zero();
  RowStream<T> a(F + ns + int64_t(c0) * N, N, w);
  RhsStream<T, NC, V, true> x(A, g.k, j0, rc, 0, N - ns <= nrows ? rows_s : rows);
  TilePipe<T, NC, true>::run(ring, N - ns, w, rc, acc, a, x);
  tile_subtract(y, acc);
  y.each(w, [&](int c, int j, T& v) {
    if (c < w && j < rc) Bo[int64_t(first + c0 + c) * g.k + j0 + j] = v;
  });
}

// ------------------------------------------------------------ permutations
template <typename TI, typename TO>
__global__ void k_perm_in(const TI* __restrict__ b, int64_t bstride,
                          const int32_t* __restrict__ perm, int n, int k,
                          TO* __restrict__ dst) {
  const int64_t total = int64_t(n) * k;
  const int bb = blockIdx.y;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = idx / k;
    const int j = static_cast<int>(idx - i * k);
    dst[int64_t(bb) * total + idx] =
        TO(b[int64_t(bb) * bstride + int64_t(perm[i]) * k + j]);
  }
}

template <typename TI, typename TO>
__global__ void k_perm_out(const TI* __restrict__ src, const int32_t* __restrict__ perm,
                           int n, int k, TO* __restrict__ x) {
  const int64_t total = int64_t(n) * k;
  const int bb = blockIdx.y;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = idx / k;
    const int j = static_cast<int>(idx - i * k);
    x[int64_t(bb) * total + int64_t(perm[i]) * k + j] =
        TO(src[int64_t(bb) * total + idx]);
  }
}

template <typename TI, typename TO>
__global__ void k_convert(const TI* __restrict__ src, int64_t sstride, int64_t count,
                          TO* __restrict__ dst) {
  const int bb = blockIdx.y;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count;
       i += int64_t(gridDim.x) * blockDim.x)
    dst[int64_t(bb) * count + i] = TO(src[int64_t(bb) * sstride + i]);
}

// ------------------------------------------------------------ refinement
// The float32 work buffers hold their right-hand sides in rows of rhs_ld(k)
// floats, k rounded up to four, the columns beyond k zero: whatever k is, the
// substitution copies and reduces 16 bytes at a time.  The kernels between
// those rows and the callers' float64 rows of k take four columns per thread;
// V = 2 where the float64 rows are 16-byte aligned, else 1.

// up to four doubles of a row whose columns from j on number `left`
template <int V>
__device__ __forceinline__ void load_quad(const double* p, int left, double (&v)[4]) {
#pragma unroll
  for (int h = 0; h < 4; h += V) {
    if constexpr (V == 2) {
      const double2 q = h < left ? *reinterpret_cast<const double2*>(p + h) : make_double2(0, 0);
      v[h] = q.x;
      v[h + 1] = q.y;
    } else {
      v[h] = h < left ? p[h] : 0.0;
    }
  }
}

// b (float64, n x k) -> buffer A of a solve: float rows of kp for float32 plans,
// double rows of kp = k for float64 ones.  nz (null: not wanted) marks, for each
// system, the supernodes that a nonzero row belongs to (sn_of) and those above
// them: the sources of a survey are a few electrodes, and the large forward
// products of every other supernode have nothing to do.  A walk upwards ends
// at a mark: whoever set that one walks on from it.  rows (null: all n of them):
// the rows to copy.
template <typename T, int V>
__global__ void k_rhs_in(const double* __restrict__ b, int64_t bstride, int n, int k, int kp,
                         T* __restrict__ rhs, const int32_t* __restrict__ rows, int nrows,
                         const int32_t* __restrict__ sn_of,
                         const int32_t* __restrict__ parent, int32_t* nz, int nsuper) {
  const int kq = kp / 4 + (kp % 4 != 0);
  const int64_t total = int64_t(nrows) * kq;
  const double* Bv = b + int64_t(blockIdx.y) * bstride;
  T* R = rhs + int64_t(blockIdx.y) * n * kp;
  volatile int32_t* mark = nz + (nz != nullptr ? int64_t(blockIdx.y) * nsuper : 0);
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t q = idx / kq, i = rows != nullptr ? rows[q] : q;
    const int j = static_cast<int>(idx - q * kq) * 4, left = k - j;
    double v[4];
    load_quad<V>(Bv + i * k + j, left, v);
    T* r = R + i * kp + j;
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(r) =
          make_float4(float(v[0]), float(v[1]), float(v[2]), float(v[3]));
    } else {
#pragma unroll
      for (int h = 0; h < 4; h += V)
        if (h < left) {
          if constexpr (V == 2)
            *reinterpret_cast<double2*>(r + h) = make_double2(v[h], v[h + 1]);
          else
            r[h] = v[h];
        }
    }
    // (a NaN is not a zero)
    if (nz != nullptr && !(v[0] == 0.0 && v[1] == 0.0 && v[2] == 0.0 && v[3] == 0.0))
      for (int s = sn_of[i]; s >= 0 && mark[s] == 0; s = parent[s]) mark[s] = 1;
  }
}

// r = b - A x in float64 (permuted order), stored as float, with max|r| and
// max|b| folded into maxbits[0..1] (the refinement state's rmax, bmax).
// Threads walk the rows in the permuted order: the nested dissection keeps
// each subdomain's rows together, and b and r move as contiguous rows (walking
// the matrix's own order measured 11 % slower on the 269,001-node benchmark).
// The pattern is kept in that order (pptr, pcol, and pent, the place of each
// entry's value), so that an x is two dependent loads away and not four.
// Measured, 56,525 nodes x 12 systems x 186 right-hand sides: 0.71 ms; one column
// per thread through perm, crow, col and iperm took 1.38 ms.
template <int V>
__global__ void k_residual(DevSym S, const double* __restrict__ vals, int64_t vals_stride,
                           const double* __restrict__ b, int64_t bstride,
                           const double* __restrict__ x, int n, int k, int kp,
                           float* __restrict__ r32, unsigned long long* __restrict__ maxbits,
                           const int* skip) {
  if (ir_skip(skip)) return;
  const int bb = blockIdx.y;
  const double* W = vals + int64_t(bb) * vals_stride;
  const double* X = x + int64_t(bb) * n * k;
  const double* Bv = b + int64_t(bb) * bstride;
  // n * k < 2^31 (checked at launch): 32-bit index arithmetic
  const int kq = kp / 4, total = n * kq;
  float4* R = reinterpret_cast<float4*>(r32) + int64_t(bb) * total;
  double rmax = 0.0, bmax = 0.0;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += gridDim.x * blockDim.x) {
    const int i = idx / kq, j = (idx - i * kq) * 4, left = k - j;
    double acc[4];
    load_quad<V>(Bv + int64_t(i) * k + j, left, acc);
#pragma unroll
    for (int h = 0; h < 4; ++h) bmax = fmax(bmax, fabs(acc[h]));
    const int e1 = S.pptr[i + 1];
#pragma unroll 4
    for (int e = S.pptr[i]; e < e1; ++e) {
      const double a = W[S.pent[e]];
      double v[4];
      load_quad<V>(X + int64_t(S.pcol[e]) * k + j, left, v);
#pragma unroll
      for (int h = 0; h < 4; ++h) acc[h] -= a * v[h];
    }
    R[idx] = make_float4(float(acc[0]), left > 1 ? float(acc[1]) : 0.f,
                         left > 2 ? float(acc[2]) : 0.f, left > 3 ? float(acc[3]) : 0.f);
#pragma unroll
    for (int h = 0; h < 4; ++h)
      if (h < left) rmax = fmax(rmax, fabs(acc[h]));
  }
  // non-negative doubles order like their bit patterns
  for (int o = 16; o > 0; o >>= 1) {
    rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
    bmax = fmax(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&maxbits[0], __double_as_longlong(rmax));
    atomicMax(&maxbits[1], __double_as_longlong(bmax));
  }
}

// x = c (first) or x += c, folding max|c| and max|x| into the refinement
// state (corrections only); rows: nbatch n of them
template <int V>
__global__ void k_ir_update(const float* __restrict__ c, int64_t rows, int k, int kp,
                            double* __restrict__ x, int first, IrState* ir) {
  if (!first && ir_skip(&ir->done)) return;
  const int kq = kp / 4;
  const int64_t total = rows * kq;
  double cmax = 0.0, xmax = 0.0;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = idx / kq;
    const int j = static_cast<int>(idx - i * kq) * 4, left = k - j;
    const float4 f = reinterpret_cast<const float4*>(c)[idx];
    const double ci[4] = {f.x, f.y, f.z, f.w};
    double* xr = x + i * k + j;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (!first) load_quad<V>(xr, left, v);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      v[h] = first ? ci[h] : v[h] + ci[h];
      if (h < left) {
        cmax = fmax(cmax, fabs(ci[h]));
        xmax = fmax(xmax, fabs(v[h]));
      }
    }
#pragma unroll
    for (int h = 0; h < 4; h += V)
      if (h < left) {
        if constexpr (V == 2)
          *reinterpret_cast<double2*>(xr + h) = make_double2(v[h], v[h + 1]);
        else
          xr[h] = v[h];
      }
  }
  if (first) return;
  for (int o = 16; o > 0; o >>= 1) {
    cmax = fmax(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
    xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
  }
  // non-negative doubles order like their bit patterns
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&ir->cmax, __double_as_longlong(cmax));
    atomicMax(&ir->xmax, __double_as_longlong(xmax));
  }
}

// zeros in the rows of the supernodes `sn` (one CTA each per system): those
// whose products accumulate
__global__ void k_clear_rows(DevSym S, const int32_t* __restrict__ sn, float* __restrict__ buf,
                             int64_t stride, int k) {
  const int s = sn[blockIdx.x];
  float4* p = reinterpret_cast<float4*>(buf + int64_t(blockIdx.y) * stride +
                                        int64_t(S.sn_first[s]) * k);
  const int64_t count = int64_t(S.sn_first[s + 1] - S.sn_first[s]) * k / 4;
  for (int64_t i = threadIdx.x; i < count; i += blockDim.x) p[i] = make_float4(0, 0, 0, 0);
}

// One thread, after correction `iter` (1-based): the estimate of the error
// of x (see IrState), the stopping decision, and DCT_ERR_IR_NOT_CONVERGED in
// the plan's status words (supernode -1, system = iterations) when the
// iterations stagnate or run out above the tolerance.  A NaN correction
// always counts as a failure; a correction at the float64 rounding level of
// x (rho <= 4 eps) ends the refinement as converged.  tol = 0 asks for a
// fixed number of corrections: a stall or running out of them then just
// ends the refinement.
__global__ void k_ir_decide(IrState* ir, int* status, unsigned long long* resid_bits,
                            int iter, int max_iters, double tol) {
  if (ir->done) return;
  // the residual of this iteration becomes the plan's reported residual
  resid_bits[0] = ir->rmax;
  resid_bits[1] = ir->bmax;
  ir->rmax = 0ull;
  ir->bmax = 0ull;
  const double c = __longlong_as_double(static_cast<long long>(ir->cmax));
  const double x = __longlong_as_double(static_cast<long long>(ir->xmax));
  const double rho = x > 0.0 ? c / x : (c > 0.0 ? INFINITY : 0.0);
  const double prev = iter > 1 ? ir->rho[min(iter - 2, kIrHistory - 1)] : 1.0;
  const double q = iter > 1 ? fmin(1.0, rho / prev) : rho;
  const double est = rho * q;
  ir->rho[min(iter - 1, kIrHistory - 1)] = rho;
  ir->iters = iter;
  ir->est = est;
  ir->cmax = 0ull;
  ir->xmax = 0ull;
  const bool nan = !(rho == rho);
  const bool floor = rho <= 4.0 * 2.220446049250313e-16;
  const bool ok = !nan && (floor || (tol > 0.0 && est <= tol));
  const bool stalled = nan || (iter > 1 && rho > 0.5 * prev);
  if (ok) {
    ir->converged = 1;
    ir->done = 1;
  } else if (stalled || iter >= max_iters) {
    // a stall at the accuracy float64 residuals allow is no error under a
    // fixed count (tol = 0); a NaN always is
    ir->done = 1;
    if ((nan || tol > 0.0) && atomicCAS(&status[0], 0, DCT_ERR_IR_NOT_CONVERGED) == 0) {
      status[1] = -1;
      status[2] = iter;
    }
  }
}

// right-hand sides per CTA of the products of the larger supernodes: the fewest columns that hold
// k, or chunks of 64 (whose fragments beyond k the double products skip)
int tile_columns(int k) { return k <= 8 ? 8 : (k <= 16 ? 16 : (k <= 32 ? 32 : 64)); }

// one launch of a substitution kind on tiles of NC right-hand sides
template <typename T, int NC>
cudaError_t launch_tiles(dct_plan* P, int kind, SolveArgs<T> g, SmallShape sh,
                         int64_t count, cudaStream_t st) {
  g.nchunk = (g.k + NC - 1) / NC;
  dim3 grid(static_cast<unsigned>(count * g.nchunk), P->nbatch);
  const dim3 block(kThreads);
  auto go = [&](auto fn, size_t smem, auto... more) {
    const cudaError_t e = allow_smem(P, fn);
    return e != cudaSuccess ? e : launch_pdl(fn, grid, block, smem, st, g, more...);
  };
  if (kind == kFwdSmall || kind == kBwdSmall) {
    sh.chunks = small_chunks<T, NC>(count * P->nbatch, sh.nb, g.nchunk);
    grid.x = static_cast<unsigned>(count * ((g.nchunk + sh.chunks - 1) / sh.chunks));
    const int in = kind == kFwdSmall ? sh.w : std::min(sh.nb, kPanel);
    const size_t smem = SmallPlaces<T, NC>(sh.w, sh.nb, in, sh.chunks > 1).bytes(sh.nb);
    auto small = [&](auto loop) {
      constexpr bool L = decltype(loop)::value;
      return kind == kFwdSmall ? go(k_fwd_small<T, NC, L>, smem, sh)
                               : go(k_bwd_small<T, NC, L>, smem, sh);
    };
    if constexpr (kSmallLoop<T, NC>)
      if (sh.chunks > 1) return small(std::true_type{});
    return small(std::false_type{});
  }
  if constexpr (sizeof(T) != 4) {
    constexpr size_t km = sizeof(T) * TilePipe<T, NC, false>::kElems;
    constexpr size_t mk = sizeof(T) * TilePipe<T, NC, true>::kElems;
    const int nrows = std::min(sh.nb, kGemmRows);
    constexpr int V = 16 / sizeof(T);
    const bool wide = sh.wide != 0;
    switch (kind) {
      case kFwdLinv: return go(wide ? k_fwd_linv<T, NC, V> : k_fwd_linv<T, NC, 1>, km);
      case kFwdBnd: return go(wide ? k_fwd_bnd<T, NC, V> : k_fwd_bnd<T, NC, 1>, km);
      case kBwdLinv: return go(wide ? k_bwd_linv<T, NC, V> : k_bwd_linv<T, NC, 1>, mk);
      case kBwdGemm:
        return go(wide ? k_bwd_gemm<T, NC, V> : k_bwd_gemm<T, NC, 1>, mk + 4 * size_t(nrows), nrows);
    }
  }
  return cudaErrorInvalidValue;
}
template <typename T>
cudaError_t launch_tiles(dct_plan* P, int kind, const SolveArgs<T>& g, SmallShape sh,
                         int64_t count, cudaStream_t st) {
  constexpr int V = 16 / sizeof(T);
  sh.wide = g.k % V == 0 && (reinterpret_cast<uintptr_t>(g.A) & 15) == 0 &&
            (reinterpret_cast<uintptr_t>(g.B) & 15) == 0 &&
            (g.b == nullptr ||
             ((reinterpret_cast<uintptr_t>(g.b) & 15) == 0 && g.bstride % V == 0));
  const bool small = kind == kFwdSmall || kind == kBwdSmall;
  switch (small ? small_columns<T>(g.k, sh.w, sh.nb) : tile_columns(g.k)) {
    case 8: return launch_tiles<T, 8>(P, kind, g, sh, count, st);
    case 16: return launch_tiles<T, 16>(P, kind, g, sh, count, st);
    case 32: return launch_tiles<T, 32>(P, kind, g, sh, count, st);
    default: return launch_tiles<T, 64>(P, kind, g, sh, count, st);
  }
}

inline dim3 grid1d(int64_t total, int ny) {
  int64_t blocks = (total + kThreads - 1) / kThreads;
  blocks = blocks < 1 ? 1 : (blocks > 148 * 16 ? 148 * 16 : blocks);
  return dim3(static_cast<unsigned>(blocks), ny);
}

// transposed: solve A^T x = b (general plans: A^T = (L U)^T = M L^T with
// M = U^T, so the forward pass runs on M and the backward pass on L)
template <typename T>
cudaError_t solve_impl(dct_plan* P, T* bufA, T* bufB, int k, cudaStream_t st,
                       bool transposed = false, bool marked = false,
                       const double* b = nullptr, int64_t bstride = 0) {
  cudaError_t e = cudaSuccess;
  SolveArgs<T> g{P->ds, nullptr, static_cast<const T*>(P->fronts), P->front_stride,
                 static_cast<const T*>(P->dinv), P->d_dinv_off, P->dinv_stride,
                 bufA, bufB, P->sym.n, k, 1, P->status,
                 static_cast<const T*>(P->linv), P->d_linv_off, P->linv_stride,
                 P->dtype == DCT_F32 && P->ir != nullptr ? &P->ir->done : nullptr,
                 marked ? P->nz : nullptr, P->sym.nsuper, nullptr, 0};
  constexpr bool kTc = sizeof(T) == 4;
  const size_t work = sizeof(T) * size_t(P->nbatch) * P->sym.n * k;
  const double nb = P->nbatch;
  // general plans: the forward pass runs on L (or M when transposed), the
  // backward pass on the other factor, each with its own inverses
  const T* fac[2] = {static_cast<const T*>(P->fronts), static_cast<const T*>(P->fronts)};
  const T* dv[2] = {static_cast<const T*>(P->dinv), static_cast<const T*>(P->dinv)};
  const T* lv[2] = {static_cast<const T*>(P->linv), static_cast<const T*>(P->linv)};
  if (P->lu) {
    const int m = transposed ? 0 : 1;   // the pass that runs on M = U^T
    fac[m] = static_cast<const T*>(P->fronts2);
    dv[m] = static_cast<const T*>(P->dinv2);
    lv[m] = static_cast<const T*>(P->linv2);
  }
  for (const Schedule* sc : {&P->fwd, &P->bwd}) {
    const int pass = sc == &P->fwd ? 0 : 1;
    g.fronts = fac[pass];
    g.dinv = dv[pass];
    g.linv = lv[pass];
    if constexpr (kTc) {
      // the rows that the tensor-core products accumulate into
      T* buf = sc == &P->fwd ? bufB : bufA;
      if (P->n_tc == P->sym.nsuper)
        e = cudaMemsetAsync(buf, 0, work, st);
      else if (P->n_tc > 0)
        k_clear_rows<<<dim3(static_cast<unsigned>(P->n_tc), P->nbatch), kThreads, 0, st>>>(
            P->ds, P->d_tc, buf, int64_t(P->sym.n) * k, k);
      if (e == cudaSuccess) e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    for (size_t li = 0; li < sc->launches.size(); ++li) {
      const Launch& L = sc->launches[li];
      if (L.count <= 0) continue;
      if ((e = P->prof.begin(L.kind, sc->flops[li] * k * nb,
                             (sc->bytes[li] + sc->bytes_rhs[li] * k) * nb, st)) !=
          cudaSuccess)
        return e;
      g.tasks = sc->d_tasks + L.first;
      if constexpr (std::is_same_v<T, double>) {
        // the first forward launch takes the rows that launch_rhs_in left out
        const bool here = pass == 0 && li == 0 && b != nullptr && P->d_inner != nullptr;
        g.b = here ? b : nullptr;
        g.bstride = bstride;
      }
      switch (L.kind) {
        case kFwdLinvTc:
        case kFwdBndTc:
        case kBwdGemmTc:
        case kBwdLinvTc:
          if constexpr (kTc) {
            e = launch_solve_tc(P, L.kind, g, L.count, st);
            if (e != cudaSuccess) return e;
            break;
          }
          return cudaErrorInvalidValue;
        default:
          // every launch of a solve but the first follows one of its own
          e = launch_tiles<T>(P, L.kind, g, SmallShape{sc->max_ns[li], sc->max_nb[li],
                                                       pass == 1 || li > 0, 0, 1},
                              L.count, st);
          if (e != cudaSuccess) return e;
      }
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      if ((e = P->prof.end(st)) != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace

// f64 plans: the permuted right-hand side is in `xa` (buffer A) and the
// solution is left there; P->bufB serves as buffer B.  b (null: all of it is in
// xa): launch_rhs_in prepared the solve, with the right-hand sides still in b,
// bstride apart for the systems.
cudaError_t run_solve_f64(dct_plan* P, double* xa, int k, cudaStream_t st,
                          bool transposed, const double* b, int64_t bstride) {
  return solve_impl<double>(P, xa, static_cast<double*>(P->bufB), k, st, transposed,
                            b != nullptr, b, bstride);
}

// complex128 plans: as float64, on complex buffers
cudaError_t run_solve_c128(dct_plan* P, cplx* xa, int k, cudaStream_t st) {
  return solve_impl<cplx>(P, xa, static_cast<cplx*>(P->bufB), k, st);
}

// f32 plans: right-hand side in P->bufA (float, A), P->bufB (B), rows of
// rhs_ld(k).
cudaError_t run_solve_f32(dct_plan* P, int k, cudaStream_t st, bool marked) {
  return solve_impl<float>(P, static_cast<float*>(P->bufA), static_cast<float*>(P->bufB),
                           rhs_ld(k), st, false, marked);
}

cudaError_t launch_perm_in_any(const void* b, int b_dtype, int64_t bstride,
                               const int32_t* perm, int n, int k, int nbatch,
                               void* dst, int dst_dtype, cudaStream_t st) {
  dim3 g = grid1d(int64_t(n) * k, nbatch);
  if (b_dtype == DCT_C128 || dst_dtype == DCT_C128) {
    if (b_dtype != dst_dtype) return cudaErrorInvalidValue;
    k_perm_in<cplx, cplx><<<g, kThreads, 0, st>>>(static_cast<const cplx*>(b), bstride, perm,
                                                  n, k, static_cast<cplx*>(dst));
    return cudaGetLastError();
  }
  if (b_dtype == DCT_F64 && dst_dtype == DCT_F64)
    k_perm_in<double, double><<<g, kThreads, 0, st>>>(
        static_cast<const double*>(b), bstride, perm, n, k, static_cast<double*>(dst));
  else if (b_dtype == DCT_F64 && dst_dtype == DCT_F32)
    k_perm_in<double, float><<<g, kThreads, 0, st>>>(
        static_cast<const double*>(b), bstride, perm, n, k, static_cast<float*>(dst));
  else if (b_dtype == DCT_F32 && dst_dtype == DCT_F64)
    k_perm_in<float, double><<<g, kThreads, 0, st>>>(
        static_cast<const float*>(b), bstride, perm, n, k, static_cast<double*>(dst));
  else
    k_perm_in<float, float><<<g, kThreads, 0, st>>>(
        static_cast<const float*>(b), bstride, perm, n, k, static_cast<float*>(dst));
  return cudaGetLastError();
}

cudaError_t launch_perm_out_any(const void* src, int src_dtype, const int32_t* perm,
                                int n, int k, int nbatch, void* x, int x_dtype,
                                cudaStream_t st) {
  dim3 g = grid1d(int64_t(n) * k, nbatch);
  if (src_dtype == DCT_C128 || x_dtype == DCT_C128) {
    if (src_dtype != x_dtype) return cudaErrorInvalidValue;
    k_perm_out<cplx, cplx><<<g, kThreads, 0, st>>>(static_cast<const cplx*>(src), perm, n, k,
                                                   static_cast<cplx*>(x));
    return cudaGetLastError();
  }
  if (src_dtype == DCT_F64 && x_dtype == DCT_F64)
    k_perm_out<double, double><<<g, kThreads, 0, st>>>(
        static_cast<const double*>(src), perm, n, k, static_cast<double*>(x));
  else if (src_dtype == DCT_F64 && x_dtype == DCT_F32)
    k_perm_out<double, float><<<g, kThreads, 0, st>>>(
        static_cast<const double*>(src), perm, n, k, static_cast<float*>(x));
  else if (src_dtype == DCT_F32 && x_dtype == DCT_F64)
    k_perm_out<float, double><<<g, kThreads, 0, st>>>(
        static_cast<const float*>(src), perm, n, k, static_cast<double*>(x));
  else
    k_perm_out<float, float><<<g, kThreads, 0, st>>>(
        static_cast<const float*>(src), perm, n, k, static_cast<float*>(x));
  return cudaGetLastError();
}

cudaError_t launch_convert_any(const void* src, int src_dtype, int64_t sstride,
                               int64_t count, int nbatch, void* dst, int dst_dtype,
                               cudaStream_t st) {
  dim3 g = grid1d(count, nbatch);
  if (src_dtype == DCT_F64 && dst_dtype == DCT_F32)
    k_convert<double, float><<<g, kThreads, 0, st>>>(
        static_cast<const double*>(src), sstride, count, static_cast<float*>(dst));
  else if (src_dtype == DCT_F64 && dst_dtype == DCT_F64)
    k_convert<double, double><<<g, kThreads, 0, st>>>(
        static_cast<const double*>(src), sstride, count, static_cast<double*>(dst));
  else if (src_dtype == DCT_F32 && dst_dtype == DCT_F64)
    k_convert<float, double><<<g, kThreads, 0, st>>>(
        static_cast<const float*>(src), sstride, count, static_cast<double*>(dst));
  else
    k_convert<float, float><<<g, kThreads, 0, st>>>(
        static_cast<const float*>(src), sstride, count, static_cast<float*>(dst));
  return cudaGetLastError();
}

// rows of k doubles can be read two at a time
static bool even_rows(const double* p, int64_t stride, int k) {
  return k % 2 == 0 && stride % 2 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

cudaError_t launch_rhs_in(dct_plan* P, const double* b, int64_t bstride, int k, void* rhs,
                          cudaStream_t st) {
  const int n = P->sym.n, nsuper = P->sym.nsuper;
  const bool f32 = P->dtype == DCT_F32;
  const int kp = f32 ? rhs_ld(k) : k;
  if (P->nz != nullptr) {
    const cudaError_t e =
        cudaMemsetAsync(P->nz, 0, sizeof(int32_t) * size_t(P->nbatch) * nsuper, st);
    if (e != cudaSuccess) return e;
  }
  const int32_t* rows = f32 ? nullptr : P->d_inner;   // float64: see run_solve_f64
  const int nrows = rows != nullptr ? P->n_inner : n;
  if (nrows == 0) return cudaSuccess;
  const dim3 g = grid1d(int64_t(nrows) * ((kp + 3) / 4), P->nbatch);
  // the copies of the float64 rows are as wide as both sides allow
  const bool even = even_rows(b, bstride, k) &&
                    (f32 || (reinterpret_cast<uintptr_t>(rhs) & 15) == 0);
  auto go = [&](auto* out, auto fn) {
    fn<<<g, kThreads, 0, st>>>(b, bstride, n, k, kp, out, rows, nrows, P->d_sn_of, P->d_parent,
                               P->nz, nsuper);
  };
  if (f32)
    go(static_cast<float*>(rhs), even ? k_rhs_in<float, 2> : k_rhs_in<float, 1>);
  else
    go(static_cast<double*>(rhs), even ? k_rhs_in<double, 2> : k_rhs_in<double, 1>);
  return cudaGetLastError();
}

cudaError_t launch_residual(dct_plan* P, const double* b, int64_t bstride,
                            const double* x, int k, cudaStream_t st) {
  const int n = P->sym.n, kp = rhs_ld(k);
  if (int64_t(n) * k >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  const int64_t nnz = static_cast<int64_t>(P->sym.nnz_in);
  auto fn = even_rows(b, bstride, k) && even_rows(x, int64_t(n) * k, k) ? k_residual<2>
                                                                        : k_residual<1>;
  fn<<<grid1d(int64_t(n) * kp / 4, P->nbatch), kThreads, 0, st>>>(
      P->ds, P->vals64, nnz, b, bstride, x, n, k, kp, static_cast<float*>(P->bufA), &P->ir->rmax,
      &P->ir->done);
  return cudaGetLastError();
}

cudaError_t launch_ir_update(dct_plan* P, double* x, int k, int first,
                             cudaStream_t st) {
  const int kp = rhs_ld(k);
  const int64_t rows = int64_t(P->nbatch) * P->sym.n;
  auto fn = even_rows(x, 0, k) ? k_ir_update<2> : k_ir_update<1>;
  fn<<<grid1d(rows * (kp / 4), 1), kThreads, 0, st>>>(static_cast<const float*>(P->bufA), rows, k,
                                                      kp, x, first, P->ir);
  return cudaGetLastError();
}

cudaError_t launch_ir_decide(dct_plan* P, int iter, cudaStream_t st) {
  k_ir_decide<<<1, 1, 0, st>>>(P->ir, P->status, P->resid_bits, iter, P->ir_iters,
                                P->ir_tol);
  return cudaGetLastError();
}

}  // namespace dct
