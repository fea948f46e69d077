// Float32 substitution products of the large supernodes on the tensor cores.
//
// Each of the four block products of the supernodal substitution is one
// launch kind of the same kernel, D (128 x N) = sum_k A[m, k] B[k, n], with
// the N right-hand sides (<= 256 per CTA) as the MMA's N dimension:
//
//   kFwdLinvTc  y_s   += L_ss^{-1}[rows m, k] b_s[k]        (B <- A rows)
//   kFwdBndTc   b_B   -= L_Bs[rows m, k] y_s[k]             (A rows, gathered)
//   kBwdGemmTc  y_s   -= L_Bs^T[cols m, k] x_B[k]           (B <- gathered A)
//   kBwdLinvTc  x_s   += L_ss^{-T}[cols m, k] y_s[k]        (A <- B rows)
//
// A task covers one 128-row tile of the output and a K range [k0, k1); every
// task adds its product into the destination rows -- one bulk f32 reduction
// per row (cp.reduce.async.bulk; k is a multiple of 4, see solve.cu) -- so K
// ranges can be split over tasks, and the destination rows of the two inverse
// products are cleared before the pass that writes them.  tcgen05.mma kind::tf32
// with the 3xTF32 split (hi*hi + hi*lo + lo*hi: Markidis et al. 2018; Ootomo
// and Yokota 2022) accumulates in TMEM.
//
// Operands move in K stages of 16.  The threads of warps 0-7 load their
// values of stage st + 1 into registers while the MMAs of stage st run, split
// them into the hi/lo operands of one of two sets in shared memory, and arrive
// at the set's "full" barrier; warp 8 issues its MMAs, whose commit is the
// set's "empty" barrier.  There is no CTA-wide barrier in the loop: with one,
// the warp whose thread issued the MMAs came late to it and the others waited.
// What bounds a stage now (about 2,000 cycles, of which its MMAs take 650 on the
// tensor pipe that two CTAs share) is the latency of its loads; a second
// register set for A, two stages ahead, gained nothing.
// Measured, five passes of the 269,001-node benchmark, 200 right-hand sides:
// 12.9 ms, with the values copied to shared memory first and two CTA-wide
// barriers per stage 14.6; 40,480 nodes, 67 right-hand sides 2.1 against 2.9.
#include <cuda_runtime.h>

#include "dct_internal.h"
#include "tc_common.cuh"

namespace dct {
namespace {

constexpr int kStK = 16;                     // K per pipeline stage
#ifndef DCT_TC_RHS
#define DCT_TC_RHS 256
#endif
#ifndef DCT_TC_CTAS_PER_SM
#define DCT_TC_CTAS_PER_SM 2
#endif
constexpr int kStN = DCT_TC_RHS;             // right-hand sides per CTA
constexpr int kNT = 256;                     // threads that load and split operands
constexpr int kTcCta = kNT + 32;             // and the warp that issues the MMAs
// split A operand (128 x 16), K-major: K-adjacent core matrices 160 B apart,
// so that the transposed stores (2 rows x 16 K per warp instruction) go to 32
// distinct banks; the natural ones (16 bytes for 8 rows at a time) do anyway.
constexpr uint32_t kALbo = 160, kASbo = (kStK / 4 - 1) * kALbo + 128;   // 608
constexpr int kABytes = (kTcM / 8) * kASbo;                             // 9728
// split B operand (16 K x 256 N), K-major: N-groups of 8 kBSbo = 528 B apart
constexpr uint32_t kBLbo = 128, kBSbo = (kStK / 4) * kBLbo + 16;       // 528
constexpr int kBBytes = (kStN / 8) * kBSbo;                            // 16896
constexpr int kSplitBytes = 2 * kABytes + 2 * kBBytes;
constexpr int kSets = 2;                     // sets of split operands
constexpr int kTcRows = kMaxSplitK;          // boundary rows of a backward task
constexpr size_t kSolveTcSmem = kSets * size_t(kSplitBytes) + kTcRows * 4 + 64;
constexpr int kCtasPerSm = DCT_TC_CTAS_PER_SM;
static_assert(kCtasPerSm * (kSolveTcSmem + 1024) <= 233472, "CTAs per SM");
static_assert(64 * (kStN + 4) * 4 <= kSets * kSplitBytes,
              "64 staged output rows fit in the operand buffers");
static_assert(kASbo % 16 == 0 && kABytes % 16 == 0 && kBSbo % 16 == 0 && kBBytes % 16 == 0,
              "descriptor alignment");

// four consecutive K values of one row -> the hi/lo operands (16 bytes each)
__device__ __forceinline__ void store_split4(unsigned char* hi, unsigned char* lo, uint32_t off,
                                             const float* v) {
  uint32_t h[4];
  float l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    h[i] = tf32_rna(v[i]);
    l[i] = v[i] - __uint_as_float(h[i]);
  }
  *reinterpret_cast<uint4*>(hi + off) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<float4*>(lo + off) = make_float4(l[0], l[1], l[2], l[3]);
}

enum TcMode { kModeFwdLinv = 0, kModeFwdBnd, kModeBwdGemm, kModeBwdLinv };

template <int MODE>
__global__ void __launch_bounds__(kTcCta, kCtasPerSm) k_solve_tc(SolveArgs<float> g) {
  constexpr bool kTrans = MODE == kModeBwdGemm || MODE == kModeBwdLinv;
  constexpr bool kInv = MODE == kModeFwdLinv || MODE == kModeBwdLinv;
  constexpr int kWarps = kNT / 32;
  static_assert(kWarps % 4 == 0, "whole warpgroups: TMEM lane quarters");
  static_assert(kNT == 256 && kStN <= kNT && kStK == 16, "the threads' shares of a stage");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int32_t* rows_s = reinterpret_cast<int32_t*>(smem_raw + kSets * kSplitBytes);
  // per split set: its operands are stored, and the MMAs that read it have
  // completed; and all MMAs have
  uint64_t* full = reinterpret_cast<uint64_t*>(rows_s + kTcRows);
  uint64_t* empty = full + kSets;
  uint64_t* done = empty + kSets;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const PanelTask tk = g.tasks[blockIdx.x];
  const int b = blockIdx.y / g.nchunk;
  const int j0 = (blockIdx.y % g.nchunk) * kStN;
  const int kc = min(kStN, g.k - j0);
  const int np = (kc + 15) & ~15;
  const DevSym& S = g.S;
  const int s = tk.s;
  const int N = S.front_n[s], first = S.sn_first[s];
  const int ns = S.sn_first[s + 1] - first;
  const int k0 = tk.p, k1 = tk.t1;
  const int m0 = tk.t0 * kTcM;
  const int32_t* rows = S.rows + S.rows_ptr[s];
  const int mvalid = min(kTcM, (MODE == kModeFwdBnd ? N - ns : ns) - m0);
  // A source: column-major, leading dimension ld; natural A[m][k] =
  // M[(roff + m) + k ld], transposed A[m][k] = M[(roff + k) + (m0 + m) ld]
  const float* M;
  int ld, roff;
  if constexpr (kInv) {
    M = g.linv + int64_t(b) * g.linv_stride + g.linv_off[s];
    ld = ns;
    roff = kTrans ? 0 : m0;
  } else {
    M = g.fronts + int64_t(b) * g.front_stride + S.front_off[s];
    ld = N;
    roff = kTrans ? ns : ns + m0;
  }
  const float* X = (MODE == kModeFwdLinv || MODE == kModeBwdGemm ? g.A : g.B) +
                   int64_t(b) * g.n * g.k;
  float* Y = (MODE == kModeFwdLinv || MODE == kModeBwdGemm ? g.B : g.A) +
             int64_t(b) * g.n * g.k;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // all of this before the wait: nothing here depends on the predecessor
  if (warp == 0) tmem_alloc(tmem_slot, kStN);
  if (tid == 0) {
    for (int q = 0; q < kSets; ++q) {
      mbar_init_n(&full[q], kWarps);
      mbar_init(&empty[q]);
    }
    mbar_init(done);
    *abort = 0;
  }
  if constexpr (MODE == kModeBwdGemm)
    for (int i = tid; i < k1 - k0; i += kTcCta) rows_s[i] = rows[ns + k0 + i];
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_wait();   // launched with launch_pdl: the predecessor's writes first
  pdl_trigger();
  const uint32_t idesc = umma_idesc_tf32(kTcM, np);
  // a finished refinement: the remaining correction launches do nothing
  bool skip = g.skip != nullptr && *reinterpret_cast<const volatile int*>(g.skip) != 0;
  // nor does the forward pass for a supernode without right-hand sides (its
  // rows of B are cleared)
  if constexpr (!kTrans) skip = skip || !rhs_reaches(g, s, b);
  const int nst = skip ? 0 : (k1 - k0 + kStK - 1) / kStK;
  // This thread's values of a stage.  Natural A: row m = tid % 128, K quads
  // tid / 128 and + 2 (a warp's loads are 32 consecutive rows); transposed A:
  // K tid % 16 of 8 rows 16 apart (a warp's loads are 16 consecutive K of two
  // rows); B: column n = tid, all 16 K (32 consecutive columns).
  constexpr int kPerA = kTcM * kStK / kNT;          // 8 values
  float ra[kPerA], rb[kStK];
  auto load_stage = [&](int st) {
    const int kb = k0 + st * kStK;
    if constexpr (kTrans) {
      const int kg = kb + (tid & 15), m = tid >> 4;
      const float* src = M + (roff + kg) + int64_t(m0 + m) * ld;
#pragma unroll
      for (int u = 0; u < kPerA; ++u) {
        bool valid = m + 16 * u < mvalid && kg < k1;
        if constexpr (MODE == kModeBwdLinv) valid = valid && kg >= m0 + m + 16 * u;
        ra[u] = valid ? __ldg(src + int64_t(16 * u) * ld) : 0.f;
      }
    } else {
      const int m = tid & 127, kq = kb + (tid >> 7) * 4;
      const float* src = M + (roff + m) + int64_t(kq) * ld;
#pragma unroll
      for (int u = 0; u < kPerA; ++u) {
        const int kg = kq + (u >> 2) * 8 + (u & 3);
        bool valid = m < mvalid && kg < k1;
        if constexpr (MODE == kModeFwdLinv) valid = valid && kg <= m0 + m;
        ra[u] = valid ? __ldg(src + int64_t((u >> 2) * 8 + (u & 3)) * ld) : 0.f;
      }
    }
    if (tid < np) {
      // plain loads: other CTAs of the chain wrote these values.  Nothing may
      // use a value here, or the loads would be waited for: a stage short of
      // K (only a task's last) takes its zeros before them.
      const float* src = X + j0 + min(tid, kc - 1);
      if (kb + kStK <= k1) {
        int row[kStK];
#pragma unroll
        for (int u = 0; u < kStK; ++u)
          row[u] = MODE == kModeBwdGemm ? rows_s[kb + u - k0] : first + kb + u;
#pragma unroll
        for (int u = 0; u < kStK; ++u) rb[u] = src[int64_t(row[u]) * g.k];
      } else {
#pragma unroll
        for (int u = 0; u < kStK; ++u) {
          rb[u] = 0.f;
          if (kb + u < k1)
            rb[u] = src[int64_t(MODE == kModeBwdGemm ? rows_s[kb + u - k0] : first + kb + u) * g.k];
        }
      }
    }
  };
  if (warp < kWarps) {
    if (nst > 0) load_stage(0);
    for (int st = 0; st < nst; ++st) {
      const int set = st % kSets;
      if (st >= kSets) {
        // the MMAs of stage st - 2, which read this stage's set (the set's
        // (st / 2 - 1)-th commit)
        int got = 1;
        if (lane == 0) got = mbar_wait_ab(&empty[set], uint32_t(st / kSets - 1) & 1u, abort);
        if (!__shfl_sync(0xffffffffu, got, 0)) break;
      }
      unsigned char* Ahi = smem_raw + set * kSplitBytes;
      unsigned char* Alo = Ahi + kABytes;
      unsigned char* Bhi = Alo + kABytes;
      unsigned char* Blo = Bhi + kBBytes;
      if constexpr (kTrans) {
        const int kl = tid & 15, m = tid >> 4;
#pragma unroll
        for (int u = 0; u < kPerA; ++u) {
          const int mu = m + 16 * u;
          tc_store_split(Ahi, Alo,
                         uint32_t(mu >> 3) * kASbo + uint32_t(kl >> 2) * kALbo +
                             uint32_t(mu & 7) * 16 + uint32_t(kl & 3) * 4,
                         ra[u]);
        }
      } else {
        const int m = tid & 127;
#pragma unroll
        for (int u = 0; u < 2; ++u)
          store_split4(Ahi, Alo,
                       uint32_t(m >> 3) * kASbo + uint32_t((tid >> 7) + 2 * u) * kALbo +
                           uint32_t(m & 7) * 16,
                       ra + 4 * u);
      }
      if (tid < np) {   // columns at or beyond np are never read
#pragma unroll
        for (int u = 0; u < kStK / 4; ++u)
          store_split4(Bhi, Blo,
                       uint32_t(tid >> 3) * kBSbo + uint32_t(u) * kBLbo + uint32_t(tid & 7) * 16,
                       rb + 4 * u);
      }
      // this warp's operands to the tensor cores
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[set]);
      if (st + 1 < nst) load_stage(st + 1);
    }
  } else if (lane == 0 && nst > 0) {
    for (int st = 0; st < nst; ++st) {
      const int set = st % kSets;
      if (!mbar_wait_ab(&full[set], uint32_t(st / kSets) & 1u, abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int kw = min(kStK, k1 - (k0 + st * kStK));
      const uint32_t ah = smem_u32(smem_raw + set * kSplitBytes), al = ah + kABytes;
      const uint32_t bh = al + kABytes, bl = bh + kBBytes;
      for (int kk = 0; kk < (kw + 7) / 8; ++kk) {
        const uint64_t dah = umma_desc(ah + kk * 2 * kALbo, kALbo, kASbo);
        const uint64_t dal = umma_desc(al + kk * 2 * kALbo, kALbo, kASbo);
        const uint64_t dbh = umma_desc(bh + kk * 2 * kBLbo, kBLbo, kBSbo);
        const uint64_t dbl = umma_desc(bl + kk * 2 * kBLbo, kBLbo, kBSbo);
        umma_tf32(tmem, dah, dbh, idesc, (st > 0 || kk > 0) ? 1u : 0u);
        umma_tf32(tmem, dah, dbl, idesc, 1u);
        umma_tf32(tmem, dal, dbh, idesc, 1u);
      }
      umma_commit(&empty[set]);
    }
    // tracks every MMA issued, also after an abort
    umma_commit(done);
  }
  // every MMA has completed (they always end, so this wait does not look at
  // the abort word); a role that gave up leaves nothing to keep
  bool ok = nst > 0;
  if (nst > 0) {
    ok = tc_wait(done, 0, g.status, DCT_ERR_DEVICE_TIMEOUT, s, b);
    if (*abort) {
      if (tid == 0) flag_timeout(g.status, s, b);
      ok = false;
    }
  }
  const float sgn = kInv ? 1.0f : -1.0f;
  // Every output row of the tile goes out as one bulk reduction
  // (cp.reduce.async.bulk .add.f32) from a staging copy in shared memory --
  // the operand buffers, free once the last MMA has completed -- instead of
  // kc / 4 vector atomics per row.
  if (ok) {
    float* stage = reinterpret_cast<float*>(smem_raw);
    // row stride: a multiple of 4 floats with stride / 4 odd, so that the
    // float4 stores of 8 consecutive rows hit distinct banks
    int ld = (kc + 3) & ~3;
    if (((ld >> 2) & 1) == 0) ld += 4;
    // all rows at once where they fit (204 right-hand sides), else two rounds
    // of 64 rows (TMEM lane quarters 2r and 2r + 1); rounds and quarters wholly
    // beyond the tile's valid rows are skipped
    const int per = kTcM * ld * 4 <= kSets * kSplitBytes ? kTcM : 64;
    for (int m1 = 0; m1 < mvalid; m1 += per) {
      const int q0 = (warp & 3) * 32;   // the quarter's first row
      if (warp < kWarps && q0 >= m1 && q0 < m1 + per && q0 < mvalid) {
        float* row = stage + (q0 - m1 + lane) * ld;
        for (int cb = (warp >> 2) * 32; cb < np; cb += (kWarps / 4) * 32) {
          uint32_t v[32];
          tmem_ld32(tmem + (uint32_t(q0) << 16) + uint32_t(cb), v);
#pragma unroll
          for (int c = 0; c < 32; c += 4)
            if (cb + c < kc)
              *reinterpret_cast<float4*>(row + cb + c) =
                  make_float4(sgn * __uint_as_float(v[c]), sgn * __uint_as_float(v[c + 1]),
                              sgn * __uint_as_float(v[c + 2]), sgn * __uint_as_float(v[c + 3]));
        }
      }
      // generic-proxy stores -> the bulk copy engine, then everyone's rows
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (tid < per) {
        const int m = m1 + tid;
        if (m < mvalid) {
          const int64_t row = MODE == kModeFwdBnd ? int64_t(rows[ns + m0 + m])
                                                  : int64_t(first + m0 + m);
          asm volatile(
              "cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(
                  Y + row * g.k + j0),
              "r"(smem_u32(stage + tid * ld)), "r"(uint32_t(kc) * 4u)
              : "memory");
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        // the staging rows are read before they are rewritten or released
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
      if (m1 + per < mvalid) __syncthreads();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kStN);
}

}  // namespace

cudaError_t launch_solve_tc(dct_plan* P, int kind, const SolveArgs<float>& g0, int64_t count,
                            cudaStream_t st) {
  if (g0.k % 4 != 0) return cudaErrorInvalidValue;
  SolveArgs<float> g = g0;
  g.nchunk = (g.k + kStN - 1) / kStN;
  const dim3 grid(static_cast<unsigned>(count), static_cast<unsigned>(P->nbatch * g.nchunk));
  auto go = [&](auto fn) {
    const cudaError_t e = allow_smem(P, fn);
    return e != cudaSuccess ? e : launch_pdl(fn, grid, dim3(kTcCta), kSolveTcSmem, st, g);
  };
  switch (kind) {
    case kFwdLinvTc: return go(k_solve_tc<kModeFwdLinv>);
    case kFwdBndTc: return go(k_solve_tc<kModeFwdBnd>);
    case kBwdGemmTc: return go(k_solve_tc<kModeBwdGemm>);
    case kBwdLinvTc: return go(k_solve_tc<kModeBwdLinv>);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace dct
