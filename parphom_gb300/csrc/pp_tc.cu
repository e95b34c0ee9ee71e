// Trailing update of the double-float reduction on the tensor cores.
//
// A(k1:n, k1:n) -= V W^H + W V^H (lower triangle) with V, W the n x jb
// panel (zlatrd, jb <= 32) in double-float, as two products X Y^H (X = V,
// Y = W, then X = W, Y = V).  Per row r each operand's 64 reals
//   [Re X(r, 0..31), Im X(r, 0..31)]
// are cut into 7 bf16 slices on a fixed-point grid set by that row's largest
// magnitude 2^E (an Ozaki-style error-free split):
//   X_r = 2^E sum_{s=0..6} 2^-8(s+1) m_s,  m_s integers, |m_0| <= 256,
//   |m_s| <= 129 for s > 0,  residual below 2^(E - 57).
// Every slice product is an integer below 2^16 and K = 64, so each sum of
// products with the same s + t (at most 2^24 in magnitude) is exact in the
// FP32 accumulation of the tensor cores.  With
//   Re(X_r Y_c^*) = ReX.ReY + ImX.ImY,   Im(X_r Y_c^*) = ImX.ReY - ReX.ImY,
// the real part pairs k-step j of the row operand with k-step j of the
// column operand and the imaginary part with k-step j ^ 2 (negated for the
// Re X half, by the instruction's negate-B bit).  The 28 slice pairs with
// s + t <= 6 go into 7 accumulators per real/imaginary part; the fold sums
// them in double-float, scales by
// 2^(E_r + E_c - 16) and subtracts from A.  Separate grids for V and W keep
// both at full relative resolution; the dropped pairs and the residual bound
// the error by about 2^-55 |X_r| |Y_c| per product, the double-float level.
//
// The tile kernel (k_cupd_tc) takes 128 rows x a few column blocks of 64, one
// CTA per SM: see there.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <cuda_bf16.h>

#include "pp_digits.cuh"
#include "pp_internal.cuh"
#include "pp_tc.cuh"

namespace pp {

namespace {

constexpr int TC_S = 7;                          // slices
constexpr int TC_KS = 4;                         // k-steps of 16 (K = 64 reals)
constexpr int TC_TILE = 4096;                    // one (slice, k-step) tile of 128 rows
constexpr int TC_OP = TC_S * TC_KS * TC_TILE;    // one operand of a 128-row block (114688)
constexpr int TC_RBLK = 2 * TC_OP;               // V and W operands of a 128-row block

// Slices of one operand row held by a warp: lane a has the complex value of
// panel column a; K index a (real part) and 32 + a (imaginary part).
template <int TILE = TC_TILE>
__device__ __forceinline__ int slice_row(zdf x, uint8_t *blk, int row, int lane) {
  float amax = fmaxf(fabsf(x.re.hi), fabsf(x.im.hi));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  int E = 0;
  if (amax > 0.f) frexpf(amax, &E);  // amax < 2^E, so |x| < 2^E
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    const df v = part ? x.im : x.re;
    const int kk = lane + 32 * part;
    float th = ldexpf(v.hi, -E), tl = ldexpf(v.lo, -E);
    uint8_t *base = blk + (kk >> 4) * TILE + tc::core_off(row, kk & 15);
#pragma unroll
    for (int s = 0; s < TC_S; ++s) {
      th = __fmul_rn(th, 256.f);
      tl = __fmul_rn(tl, 256.f);
      const float mi = rintf(th);
      two_sum(__fsub_rn(th, mi), tl, th, tl);
      *(__nv_bfloat16 *)(base + s * TC_KS * TILE) = __float2bfloat16_rn(mi);
    }
  }
  return E;
}

// Source rows of one operand: element (row, a) of matrix b is
// P[b * sP + (rbase + row) * rs + a * cs] (conjugated when conj), zero for
// a >= min(jb, n_b - 1 - k0) and, with vmask, for rbase + row < k0 + a + 1
// (the zero part of a Householder panel).  Rows 0 .. nrows_b - 1 exist, with
// nrows_b = n_b - rbase (nrows_fixed == 0) or nrows_fixed.
struct TcSliceSrc {
  const zdf *P;
  int64_t sP, rs, cs;
  int rbase, nrows_fixed, vmask, conj;
};

// Slices of rows 0 .. 128 ceil(nrows_b / 128) - 1 (rows past nrows_b are
// zero): one warp per row.  Row r of matrix b goes to block r / 128 of
// S + b sS (blocks blk bytes apart), its exponent to E[b sE + r es + eo].
__global__ void __launch_bounds__(128) k_tc_slices(TcSliceSrc src, const int *nvec, int k0, int jb, uint8_t *S,
                                                   int64_t sS, int64_t blk, int *E, int64_t sE, int es, int eo) {
  const int b = blockIdx.y;
  const int n = nvec[b];
  const int nrows = src.nrows_fixed > 0 ? src.nrows_fixed : n - src.rbase;
  if (nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rl = blockIdx.x * 4 + warp;
  if (rl >= (nrows + 127) / 128 * 128) return;
  const int jmax = min(jb, n - 1 - k0);
  zdf v{{0.f, 0.f}, {0.f, 0.f}};
  if (rl < nrows && lane < jmax && (!src.vmask || src.rbase + rl >= k0 + lane + 1)) {
    v = src.P[b * src.sP + (int64_t)(src.rbase + rl) * src.rs + (int64_t)lane * src.cs];
    if (src.conj) v.im = df_neg(v.im);
  }
  uint8_t *blkp = S + b * sS + (int64_t)(rl >> 7) * blk;
  const int e = slice_row(v, blkp, rl & 127, lane);
  if (lane == 0) E[b * sE + (int64_t)rl * es + eo] = e;
}

// One operand of a product C -= X Y^H: slices in 128-row blocks of TC_OP
// bytes placed blk bytes apart (matrix b at S + b sS), and the exponent of
// row r at E[b sE + r es + eo].
struct TcOperand {
  const uint8_t *S;
  int64_t sS, blk;
  const int *E;
  int64_t sE;
  int es, eo;
};
// C(rbase + r, cbase + c) -= sum_p X_p(r, :) Y_p(c, :)^H over the tiles of
// 128 rows x 64 columns of rows [0, nrows_b) and columns [0, ncols_b): all of
// them, or (tri) the lower triangle of a square trailing block.
struct TcUpdate {
  zdf *C;
  int64_t ldc, sC;
  int rbase, cbase;
  int ncols_fixed;  // columns: ncols_fixed, or n_b - cbase when 0; rows: n_b - rbase
  int tri, nprod;
  int cbs;  // column blocks per CTA
  TcOperand x[2], y[2];
  // test hook (pp_debug_stall_tc_wait): matrix stall_b's first CTA waits,
  // before its first row-operand wait, on an mbarrier that nothing arrives
  // on, for stall_cycles SM clocks, and so takes the time-out path; -1: off
  int stall_b;
  long long stall_cycles;
};
// CTA = 128 rows x up to cbs column blocks of 64, both products in turn.  One
// warp issues the MMAs, one copies, 16 fold:
//  * the seven groups of equal slice-index sum are formed one after the other,
//    each in one of two tensor-memory buffers (64 real + 64 imaginary columns),
//    so that the MMAs of the next groups, and of the next column block, run
//    while the warps add a finished group to their double-float sums (a
//    thread: one row, 16 columns).  Order 6, 5, 4, 0, 1, 2, 3 (fold_group):
//    long groups first, so that the end of a tile runs under them;
//  * the row operand goes through the column buffers to tensor memory once per
//    product (tcgen05.cp), which halves the shared-memory reads of an MMA:
//    32.4 cycles per 128 x 64 x 16 against 48.5 with both operands in shared
//    memory (the tensor cores' own rate: 32);
//  * the tile of C arrives in shared memory (cp.async, a thread's own elements)
//    during the MMAs.
// Per tile and product: 7.2k cycles of MMA, 8k of fold, 6.5k for the update of
// C, of which the last two are not overlapped: L2 traffic (256 KB of C, 56 KB
// of operand) and the fold's issue slots bound it now.  The earlier kernel (128
// x 32 tiles, all 14 accumulators at once, MMAs issued by lane 0, then the
// fold): n = 4764, 8 matrices, 196 ms of trailing updates and 78 ms of X -= V Y;
// now 95 and 43 ms.  (Four accumulator buffers and the row operand in shared
// memory: 167 and 68, of which the issue by lane 0 cost 62 and 26.)
constexpr int CU_N = 64;                            // columns of a block
constexpr int CU_BB = TC_S * TC_KS * CU_N * 32;     // its operand (57344 bytes)
constexpr int CU_EW = 16;                           // folding warps
constexpr int CU_NT = 32 * CU_EW + 128;             // and the issuing warpgroup (one warp works)
constexpr int CU_Q = CU_N / (CU_EW / 4);            // columns per thread (16)
constexpr int CU_ACC = 2;                           // accumulator buffers
constexpr int CU_TA = CU_ACC * 2 * CU_N;            // tensor-memory column of the row operand
constexpr int CU_CS = 14;                           // its columns of C staged in shared memory
constexpr int CU_STC = CU_CS * 32 * CU_EW * 16;     // (114688 bytes)
constexpr int CU_SMEM = TC_OP + CU_STC + 256;
static_assert(2 * CU_BB == TC_OP, "the row operand passes through the column buffers");
constexpr uint32_t CU_ID = tc::idesc_bf16(128, CU_N, 0);
constexpr uint32_t CU_IDN = tc::idesc_bf16(128, CU_N, 1);
static_assert(CU_TA + TC_S * TC_KS * 8 <= 512, "accumulators and row operand exceed tensor memory");

// Wait for a phase, giving up after `cycles` SM clocks or when another warp of
// the CTA has given up.
__device__ __forceinline__ bool wait_phase(uint64_t *bar, uint32_t parity, volatile int *abort,
                                           long long cycles = 1000000000LL) {
  const long long t0 = clock64();
  while (!tc::mbar_try(bar, parity)) {
    if (*abort || clock64() - t0 > cycles) return false;
  }
  return true;
}

// MMAs of the group u: re acc pairs row k-step j with column k-step j, im acc
// with column k-step j ^ 2, negated for j < 2 (Re X . Im Y).  A descriptor
// differs from the operand's first only in its start address (bits 0-13, in
// 16-byte units).
template <int U>
__device__ __forceinline__ void cu_issue(uint32_t tm, uint32_t ta, uint64_t b0) {
#pragma unroll
  for (int s = 0; s <= U; ++s) {
    const int t = U - s;
#pragma unroll
    for (int j = 0; j < TC_KS; ++j) {
      const uint32_t acc = (s == 0 && j == 0) ? 0u : 1u;
      const uint32_t ad = ta + (s * TC_KS + j) * 8;
      const uint64_t br = b0 + (uint64_t)((t * TC_KS + j) * (CU_N * 32 >> 4));
      const uint64_t bi = b0 + (uint64_t)((t * TC_KS + (j ^ 2)) * (CU_N * 32 >> 4));
      tc::mma_bf16_ta(tm, ad, br, CU_ID, acc);
      tc::mma_bf16_ta(tm + CU_N, ad, bi, j < 2 ? CU_IDN : CU_ID, acc);
    }
  }
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid ? 8 : 0) : "memory");
}

struct CuBars {
  uint64_t row, row_free, col[2], col_free[2], acc[CU_ACC], acc_free[CU_ACC], never, drain;
  uint32_t tmem;
  int abort;
};
static_assert(sizeof(CuBars) <= 256, "barriers fit the shared memory set aside");

__global__ void __launch_bounds__(CU_NT, 1) k_cupd_tc(TcUpdate u, const int *nvec, int *err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sBop = smem;                // two column-operand buffers
  zdf *stC = (zdf *)(smem + TC_OP);    // tile of C: 16 B per fold thread and column
  CuBars &bar = *(CuBars *)(smem + TC_OP + CU_STC);
  const int b = blockIdx.z, R = blockIdx.y, q = blockIdx.x;
  const int n = nvec[b];
  const int nrows = n - u.rbase;
  const int ncols = u.ncols_fixed > 0 ? u.ncols_fixed : n - u.cbase;
  if (nrows <= 0 || ncols <= 0) return;
  const int nrb = (nrows + 127) / 128, ncb = (ncols + CU_N - 1) / CU_N;
  if (R >= nrb) return;
  const int cb_beg = q * u.cbs;
  int cb_end = min(cb_beg + u.cbs, ncb);
  if (u.tri) cb_end = min(cb_end, 128 / CU_N * (R + 1));
  if (cb_beg >= cb_end) return;
  // an earlier wait of this matrix gave up: its results are already invalid
  if (__syncthreads_or(*(volatile int *)&err[b])) return;
  const int ncbw = cb_end - cb_beg;
  const int nblk = u.nprod * ncbw;  // (product, column block) steps

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == CU_EW) tc::tmem_alloc(&bar.tmem, 512);
  if (tid == 0) {
    tc::mbar_init(&bar.row, 1);
    tc::mbar_init(&bar.row_free, 1);
    for (int k = 0; k < 2; ++k) {
      tc::mbar_init(&bar.col[k], 1);
      tc::mbar_init(&bar.col_free[k], 1);
    }
    for (int k = 0; k < CU_ACC; ++k) {
      tc::mbar_init(&bar.acc[k], 1);
      tc::mbar_init(&bar.acc_free[k], CU_EW);
    }
    tc::mbar_init(&bar.never, 1);
    tc::mbar_init(&bar.drain, 1);
    bar.abort = 0;
    tc::mbar_init_fence();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tm = __shfl_sync(0xffffffffu, bar.tmem, 0);
  volatile int *abort = &bar.abort;
  // launched with 96 registers a thread (61440): 512 x 104 + 128 x 56 = 60416
  if (warp >= CU_EW) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    const bool one = tc::elect_one();
    bool ok = true;
    auto wait = [&](uint64_t *w, int phase, long long cycles = 1000000000LL) {
      ok = __all_sync(0xffffffffu, ok && wait_phase(w, (uint32_t)(phase & 1), abort, cycles));
    };
    if (warp == CU_EW) {
      // ---- MMAs
      const uint64_t a0 = tc::sdesc(tc::smem_u32(sBop), 128, 256);
      if (b == u.stall_b && R == 0 && q == 0) wait(&bar.never, 0, u.stall_cycles);
      for (int i = 0; i < nblk && ok; ++i) {
        const int buf = i & 1;
        if (i % ncbw == 0) {  // (the last product's MMAs have ended: the copy waited for them)
          wait(&bar.row, i / ncbw);
          if (!ok) break;
          tc::fence_after();
          if (one) {
            for (int sj = 0; sj < TC_S * TC_KS; ++sj)
              tc::tmem_cp_kstep(tm + CU_TA + sj * 8, a0 + (uint64_t)(sj * (TC_TILE >> 4)));
            tc::mma_commit(&bar.row_free);
          }
          __syncwarp();
        }
        wait(&bar.col[buf], i >> 1);
        const uint64_t b0 = tc::sdesc(tc::smem_u32(sBop + buf * CU_BB), 128, 256);
        int g = i * TC_S;
        auto group = [&](auto issue) {
          const int slot = g & (CU_ACC - 1);
          if (g >= CU_ACC) wait(&bar.acc_free[slot], g / CU_ACC - 1);
          tc::fence_after();
          if (ok && one) {
            issue(tm + slot * (2 * CU_N));
            tc::mma_commit(&bar.acc[slot]);
          }
          __syncwarp();
          ++g;
        };
        group([&](uint32_t d) { cu_issue<6>(d, tm + CU_TA, b0); });
        group([&](uint32_t d) { cu_issue<5>(d, tm + CU_TA, b0); });
        group([&](uint32_t d) { cu_issue<4>(d, tm + CU_TA, b0); });
        group([&](uint32_t d) { cu_issue<0>(d, tm + CU_TA, b0); });
        group([&](uint32_t d) { cu_issue<1>(d, tm + CU_TA, b0); });
        group([&](uint32_t d) { cu_issue<2>(d, tm + CU_TA, b0); });
        group([&](uint32_t d) { cu_issue<3>(d, tm + CU_TA, b0); });
        if (ok && one) tc::mma_commit(&bar.col_free[buf]);
        __syncwarp();
      }
      // every MMA has ended before the tensor memory is released
      if (ok) wait(&bar.col_free[(nblk - 1) & 1], (nblk - 1) >> 1);
      if (!ok) {
        // give up: tell the other warps, then let the MMAs in flight finish
        // (bounded) before the memory is released
        if (one) {
          *abort = 1;
          atomicExch(&err[b], 1);
          tc::mma_commit(&bar.drain);
          tc::mbar_wait(&bar.drain, 0u, 200000000LL);
        }
        __syncwarp();
      }
    } else if (warp == CU_EW + 1) {
      // ---- copies: the row operand through both column buffers, then its columns
      int nrow = 0, ncol = 0;  // operands requested
      auto copy_col = [&](int i) {  // column operand of step i (product i / ncbw)
        if (one) {
          const TcOperand &y = u.y[i / ncbw];
          const int cb = cb_beg + i % ncbw, buf = i & 1;
          tc::mbar_expect_tx(&bar.col[buf], CU_BB);
          const uint8_t *src = y.S + b * y.sS + (int64_t)(cb / 2) * y.blk + (cb & 1) * (CU_N * 32);
          for (int sj = 0; sj < TC_S * TC_KS; ++sj)
            tc::bulk_g2s(sBop + buf * CU_BB + sj * (CU_N * 32), src + sj * TC_TILE, CU_N * 32, &bar.col[buf]);
        }
        ++ncol;
      };
      for (int i = 0; i < nblk && ok; ++i) {
        const bool first = i % ncbw == 0, next = (i + 1) % ncbw != 0;
        if (i > 0 && (first || next)) wait(&bar.col_free[(i - 1) & 1], (i - 1) >> 1);  // step i - 1's MMAs have ended
        if (first && ok) {
          if (one) {
            const TcOperand &x = u.x[i / ncbw];
            tc::mbar_expect_tx(&bar.row, TC_OP);
            tc::bulk_g2s(sBop, x.S + b * x.sS + (int64_t)R * x.blk, TC_OP, &bar.row);
          }
          ++nrow;
          wait(&bar.row_free, i / ncbw);
          if (ok) copy_col(i);
        }
        if (next && ok) copy_col(i + 1);
        __syncwarp();
      }
      // no copy may land after the block's end
      if (nrow > 0) tc::mbar_wait(&bar.row, (uint32_t)((nrow - 1) & 1), 200000000LL);
      for (int k = max(0, ncol - 2); k < ncol; ++k) tc::mbar_wait(&bar.col[k & 1], (uint32_t)((k >> 1) & 1), 200000000LL);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ---- fold: this thread's row (= TMEM lane) and CU_Q columns of each block
    zdf *C = u.C + b * u.sC;
    const int lg = warp & 3, c0q = (warp >> 2) * CU_Q;
    const int rl = 128 * R + 32 * lg + lane;  // row within the block of rows
    const int r = u.rbase + rl;
    const uint32_t lane_addr = tm + ((uint32_t)(32 * lg) << 16) + c0q;
    bool ok = true;
    for (int i = 0; i < nblk && ok; ++i) {
      const int p = i / ncbw, cb = cb_beg + i % ncbw;
      const int cl0 = CU_N * cb + c0q;  // first column (local) of this thread
      zdf *Cr = C + r + u.ldc * (u.cbase + cl0);
      const int left = rl < nrows ? min(ncols, u.tri ? r - u.cbase + 1 : ncols) - cl0 : 0;  // columns of this thread
      if (p > 0 && i % ncbw == 0) __threadfence();  // the previous product's sums are read back below
#pragma unroll
      for (int k = 0; k < CU_CS; ++k)
        if (k < left) cp_async16(&stC[k * (32 * CU_EW) + tid], Cr + u.ldc * k, true);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const TcOperand &x = u.x[p], &y = u.y[p];
      const int er = x.E[b * x.sE + (int64_t)rl * x.es + x.eo] - 16;
      const int ecl = y.E[b * y.sE + (int64_t)(cl0 + (lane & (CU_Q - 1))) * y.es + y.eo];  // of column lane & 15
      df sr[CU_Q], si[CU_Q];
      int g = i * TC_S;
      auto fold = [&](auto add) {
        const int slot = g & (CU_ACC - 1);
        ok = __all_sync(0xffffffffu, ok && wait_phase(&bar.acc[slot], (uint32_t)((g / CU_ACC) & 1), abort));
        if (ok) {
          tc::fence_after();
#pragma unroll
          for (int c4 = 0; c4 < CU_Q; c4 += 4) {
            float re[4], im[4];
            tc::tmem_ld4(lane_addr + slot * (2 * CU_N) + c4, re);
            tc::tmem_ld4(lane_addr + slot * (2 * CU_N) + CU_N + c4, im);
            tc::tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 4; ++k) add(c4 + k, re[k], im[k]);
          }
          tc::fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&bar.acc_free[slot]);
        }
        ++g;
      };
      fold([&](int k, float x, float y) { fold_group<6>(sr[k], x); fold_group<6>(si[k], y); });
      fold([&](int k, float x, float y) { fold_group<5>(sr[k], x); fold_group<5>(si[k], y); });
      fold([&](int k, float x, float y) { fold_group<4>(sr[k], x); fold_group<4>(si[k], y); });
      fold([&](int k, float x, float y) { fold_group<0>(sr[k], x); fold_group<0>(si[k], y); });
      fold([&](int k, float x, float y) { fold_group<1>(sr[k], x); fold_group<1>(si[k], y); });
      fold([&](int k, float x, float y) { fold_group<2>(sr[k], x); fold_group<2>(si[k], y); });
      fold([&](int k, float x, float y) { fold_group<3>(sr[k], x); fold_group<3>(si[k], y); });
      if (!ok) break;
      zdf cd[CU_Q - CU_CS];
#pragma unroll
      for (int k = CU_CS; k < CU_Q; ++k)
        if (k < left) cd[k - CU_CS] = Cr[u.ldc * k];
      asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
      for (int k = 0; k < CU_Q; ++k) {
        const float sc = pow2f(er + __shfl_sync(0xffffffffu, ecl, k));
        if (k >= left) continue;
        const zdf cv = k < CU_CS ? stC[k * (32 * CU_EW) + tid] : cd[max(k - CU_CS, 0)];
        const df pr = fold_done(sr[k]), pi = fold_done(si[k]);
        Cr[u.ldc * k] = zdf{df_sub(cv.re, df{__fmul_rn(pr.hi, sc), __fmul_rn(pr.lo, sc)}),
                            df_sub(cv.im, df{__fmul_rn(pi.hi, sc), __fmul_rn(pi.lo, sc)})};
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!ok && lane == 0) {
      *abort = 1;
      atomicExch(&err[b], 1);
    }
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == CU_EW) tc::tmem_dealloc(tm, 512);
}

// Long-K products on the tensor cores over column-major DF matrices read
// row-wise: element (c, r) of A at A[r + lda c], element (j, r) of B at
// Bm[r + ldb j].
//   mode 0 (V^H X of the back-transform): C(c, j) = sum_r A(c, r) conj(B(j, r)),
//     j = the 32 panel columns (zero above the Householder unit diagonals), the
//     rows split over gridDim.y ranges, written to split-K slots of out
//     (out[(y 32 + j) ldo + c]);
//   mode 1 (E_b = X^H Z): A = Z (real, rows c < m_b: the eigenvector index),
//     C(c, j) = sum_r A(c, r) conj(B(j, r)), B = X (rows j < nrows_b: the
//     boundary row), written to out[j + ldo c].
// Exact slice products need K <= 64 reals, so the rows r are taken in chunks:
// 32 rows (re and im) in mode 0, 64 rows of the real A in mode 1.
struct LongK {
  const zdf *A;
  int64_t lda, sA;
  const zdf *Bm;
  int64_t ldb, sB;
  int nrows_b;         // mode 1: valid B rows
  int k0, jb;          // mode 0: panel k0 of width jb
  const uint8_t *S;    // mode 0: slices of B, LK_BOP bytes per chunk, and their exponents (32 per chunk)
  int64_t sS;
  const int *Ex;
  int64_t sEx;
  int rbeg;            // rows [rbeg, n_b)
  int ncols_a;         // mode 0: rows c < ncols_a
  const int64_t *rng;  // mode 1: rows c < rng[8 b + 2]
  zdf *out;
  int64_t ldo, sO;
};

constexpr int LK_BOP = TC_S * TC_KS * 1024;  // 32 rows of one operand (28672 bytes)
constexpr int LK_LD = 33;                    // staging row stride (16-byte elements)
constexpr int LK_LDB = 65;                   // and of B in mode 1
constexpr int LK_CW = 16;                    // computing warps
constexpr int LK_LW = 3;                     // loading warps
constexpr int LK_NT = 32 * (LK_CW + 1 + LK_LW);  // and the issuing one
constexpr int LK_ACC = 4;                    // accumulator buffers of 64 columns
constexpr int LK_TA = LK_ACC * 64;           // tensor-memory column of A
constexpr uint32_t LK_ID = tc::idesc_f16(128, 32, 0);
constexpr uint32_t LK_IDN = tc::idesc_f16(128, 32, 1);
static_assert(LK_TA + TC_S * TC_KS * 8 <= 512, "accumulators and A exceed tensor memory");
template <int MODE>
constexpr int lk_smem() {
  return (MODE ? 4 : 2) * LK_BOP + 128 * LK_LD * 16 + (MODE ? 32 * LK_LDB * 16 : 0) + 1024;
}
// Slices of the 32 panel columns for mode 0: chunk x (rows rbeg + 32 x ...) of
// matrix y, once per panel instead of once per 128 rows of A.
__global__ void __launch_bounds__(128) k_longk_bslice(LongK p, const int *nvec, uint8_t *S, int *Ex) {
  __shared__ zdf st[32 * LK_LD];
  const int b = blockIdx.y, n = nvec[b], tid = threadIdx.x, lane = tid & 31;
  const int r0 = p.rbeg + 32 * blockIdx.x;
  if (r0 >= n) return;
  const int nj = min(p.jb, n - 1 - p.k0);
  for (int j = tid >> 5; j < 32; j += 4) {
    const int r = r0 + lane;
    st[j * LK_LD + lane] = r < n && j < nj && r >= p.k0 + j + 1 ? p.Bm[b * p.sB + r + p.ldb * j]
                                                                 : zdf{{0.f, 0.f}, {0.f, 0.f}};
  }
  __syncthreads();
  const int j = tid >> 2, ks = tid & 3, part = ks >> 1, rb = 16 * (ks & 1);
  df x[16];
  float amax = 0.f;
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    x[t] = ((const df *)&st[j * LK_LD + rb + t])[part];
    amax = max_abs(amax, x[t].hi);
  }
  amax = max_abs(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = max_abs(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  const int E = grid_exp(amax);
  Fixed56 f[16];
  to_fixed<16>(x, E, false, f);
  uint8_t *dst = S + b * p.sS + (int64_t)blockIdx.x * LK_BOP + ks * 1024 + tc::core_off(j, 0);
  auto put = [&](auto dig, int s) {
    uint32_t w[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) w[t] = dig(f[2 * t], f[2 * t + 1]);
    *(uint4 *)(dst + s * TC_KS * 1024) = make_uint4(w[0], w[1], w[2], w[3]);
    *(uint4 *)(dst + s * TC_KS * 1024 + 128) = make_uint4(w[4], w[5], w[6], w[7]);
  };
  put([](Fixed56 a, Fixed56 c) { return digit2<0>(a, c); }, 0);
  put([](Fixed56 a, Fixed56 c) { return digit2<1>(a, c); }, 1);
  put([](Fixed56 a, Fixed56 c) { return digit2<2>(a, c); }, 2);
  put([](Fixed56 a, Fixed56 c) { return digit2<3>(a, c); }, 3);
  put([](Fixed56 a, Fixed56 c) { return digit2<4>(a, c); }, 4);
  put([](Fixed56 a, Fixed56 c) { return digit2<5>(a, c); }, 5);
  put([](Fixed56 a, Fixed56 c) { return digit2<6>(a, c); }, 6);
  if (ks == 0) Ex[b * p.sEx + 32 * (int)blockIdx.x + j] = E;
}

// MMAs of the group U.  Mode 0: as cu_issue, N = 32.  Mode 1: the real A's
// k-step with the same k-step of Re B and of Im B (an operand each).
template <int U, int MODE>
__device__ __forceinline__ void lk_issue(uint32_t d, uint32_t ta, uint64_t b0) {
#pragma unroll
  for (int s = 0; s <= U; ++s) {
    const int t = U - s;
#pragma unroll
    for (int j = 0; j < TC_KS; ++j) {
      const uint32_t acc = (s == 0 && j == 0) ? 0u : 1u;
      const uint32_t ad = ta + (s * TC_KS + j) * 8;
      const uint64_t br = b0 + (uint64_t)((t * TC_KS + j) * (1024 >> 4));
      const uint64_t bi = b0 + (uint64_t)(MODE ? ((TC_S + t) * TC_KS + j) * (1024 >> 4) : (t * TC_KS + (j ^ 2)) * (1024 >> 4));
      tc::mma_bf16_ta(d, ad, br, LK_ID, acc);
      tc::mma_bf16_ta(d + 32, ad, bi, MODE == 0 && j < 2 ? LK_IDN : LK_ID, acc);
    }
  }
}

struct LkBars {
  uint64_t b[2], done, a_ready, acc[LK_ACC], acc_free[LK_ACC], drain, st_full, st_free;
  uint32_t tmem;
  int abort;
};
static_assert(sizeof(LkBars) <= 128, "barriers fit the shared memory set aside");

// CTA = 128 rows c x 32 columns j (re and im: 64 accumulator columns).  16
// warps compute, one issues the MMAs, three load; per chunk, for the groups of
// equal slice-index sum u = 6 ... 0: a computing warp adds the finished group
// of chunk k to its double-float sums and then writes slice u of chunk k + 1 to
// tensor memory (slice u of A is read by the groups >= u only, so it is free by
// then).  The MMAs of chunk k + 1 run while the warps scale and add chunk k to
// the result and cut the grid integers of chunk k + 2.  A thread has one row
// c, 16 of its 64 reals of a chunk as 56-bit integers, and 8 columns j of the
// sums.  Instruction issue bounds it: 1440 instructions per warp and chunk, 60%
// of the issue slots (tensor cores 30%); 10.7k cycles per chunk in mode 0 and
// 15k (twice the rows) in mode 1.  The earlier kernel cut the panel anew for
// every 128 rows, with a float per digit, kept the slices of A in shared memory
// and alternated slicing, MMAs and fold: 21.6k cycles per chunk.  n = 4764, 8
// matrices: V^H X 94 -> 52 ms, X^H Z 80 -> 47 ms; n = 2604 with all vectors:
// V^H X 29.7 -> 17.3 ms.
template <int MODE>
__global__ void __launch_bounds__(LK_NT, 1) k_longk_tc(LongK p, const int *nvec, int *err) {
  constexpr int CR = MODE ? 64 : 32;  // rows r per chunk
  constexpr int BOP = (MODE ? 2 : 1) * LK_BOP;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sBop = smem;                                   // two buffers: B of a chunk, sliced
  zdf *stA = (zdf *)(smem + 2 * BOP);                     // chunk of A: row c at stA + c LK_LD
  zdf *stB = stA + 128 * LK_LD;                           // mode 1: chunk of B, row j at stB + j LK_LDB
  __shared__ float sRow[2][4 * 128];                      // largest magnitudes, [chunk & 1][k-step][row]
  __shared__ float sCol[2][16 * 32];                      // mode 1: of B, [chunk & 1][rows r][column]
  LkBars &bar = *(LkBars *)(stB + (MODE ? 32 * LK_LDB : 0));
  const int b = blockIdx.z;
  const int n = nvec[b];
  // mode 1 walks the 32-row B tiles fastest (blockIdx.x), so that the CTAs
  // sharing one 128-row tile of Z run together and read it once from DRAM
  const int ta = MODE ? blockIdx.y : blockIdx.x, tb = MODE ? blockIdx.x : 0;
  const int c0 = ta * 128;
  const int na = MODE ? (int)p.rng[b * 8 + 2] : p.ncols_a;  // valid rows c
  if (c0 >= na) return;
  const int j0 = 32 * tb;
  const int nj = MODE ? p.nrows_b : min(p.jb, n - 1 - p.k0);  // valid rows j
  if (MODE && j0 >= nj) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // chunks of CR rows r: [kc_beg, kc_beg + nk)
  const int nck = n > p.rbeg ? (n - p.rbeg + CR - 1) / CR : 0;
  const int ns = MODE ? 1 : gridDim.y, si = MODE ? 0 : blockIdx.y;
  const int kc_beg = (int)((int64_t)nck * si / ns);
  // nothing once a wait of this matrix has given up: its results are invalid
  const int nk = __syncthreads_or(*(volatile int *)&err[b]) ? 0 : (int)((int64_t)nck * (si + 1) / ns) - kc_beg;
  const int lg = warp & 3, ks = warp >> 2;
  const int cl = 32 * lg + lane;  // row c of this thread (TMEM lane)
  auto write = [&](const df *v) {  // this thread's row c and its 8 columns j
    if (c0 + cl >= na) return;
    zdf *out = p.out + b * p.sO;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int j = 8 * ks + t;
      if (MODE == 0)
        out[((int64_t)blockIdx.y * 32 + j) * p.ldo + c0 + cl] = zdf{v[t], v[8 + t]};
      else if (j0 + j < nj)
        out[j0 + j + p.ldo * (int64_t)(c0 + cl)] = zdf{v[t], v[8 + t]};
    }
  };
  if (nk > 0) {
    if (warp == LK_CW) tc::tmem_alloc(&bar.tmem, 512);
    if (tid == 0) {
      for (int k = 0; k < 2; ++k) tc::mbar_init(&bar.b[k], 1);
      tc::mbar_init(&bar.done, 1);
      tc::mbar_init(&bar.a_ready, LK_CW);
      for (int k = 0; k < LK_ACC; ++k) {
        tc::mbar_init(&bar.acc[k], 1);
        tc::mbar_init(&bar.acc_free[k], LK_CW);
      }
      tc::mbar_init(&bar.drain, 1);
      tc::mbar_init(&bar.st_full, 32 * LK_LW);
      tc::mbar_init(&bar.st_free, LK_CW);
      bar.abort = 0;
      tc::mbar_init_fence();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tm = __shfl_sync(0xffffffffu, bar.tmem, 0);
    volatile int *abort = &bar.abort;
    bool ok = true;
    // launched with 96 registers a thread (61440): 512 x 104 + 128 x 56 = 60416
    if (warp >= LK_CW) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
      const bool one = tc::elect_one();
      auto wait = [&](uint64_t *w, int phase) {
        ok = __all_sync(0xffffffffu, ok && wait_phase(w, (uint32_t)(phase & 1), abort));
      };
      int ncopy = 0;
      auto copy_b = [&](int k) {
        if (MODE == 0 && one) {
          tc::mbar_expect_tx(&bar.b[k & 1], LK_BOP);
          tc::bulk_g2s(sBop + (k & 1) * LK_BOP, p.S + b * p.sS + (int64_t)(kc_beg + k) * LK_BOP, LK_BOP, &bar.b[k & 1]);
        }
        ++ncopy;
      };
      const int nkw = warp == LK_CW ? nk : 0;
      if (nkw > 0) copy_b(0);
      if (nkw > 1) copy_b(1);
      for (int k = 0; k < nkw && ok; ++k) {
        if (MODE == 0) wait(&bar.b[k & 1], k >> 1);
        wait(&bar.a_ready, k);
        const uint64_t b0 = tc::sdesc(tc::smem_u32(sBop + (k & 1) * BOP), 128, 256);
        int g = k * TC_S;
        auto group = [&](auto issue) {
          const int slot = g & (LK_ACC - 1);
          if (g >= LK_ACC) wait(&bar.acc_free[slot], g / LK_ACC - 1);
          tc::fence_after();
          if (ok && one) {
            issue(tm + slot * 64);
            tc::mma_commit(&bar.acc[slot]);
          }
          __syncwarp();
          ++g;
        };
        group([&](uint32_t d) { lk_issue<6, MODE>(d, tm + LK_TA, b0); });
        if (k >= 1) {  // chunk k - 1's MMAs have ended: its buffer takes chunk k + 1
          wait(&bar.done, k - 1);
          if (ok && k + 1 < nk) copy_b(k + 1);
          __syncwarp();
        }
        group([&](uint32_t d) { lk_issue<5, MODE>(d, tm + LK_TA, b0); });
        group([&](uint32_t d) { lk_issue<4, MODE>(d, tm + LK_TA, b0); });
        group([&](uint32_t d) { lk_issue<3, MODE>(d, tm + LK_TA, b0); });
        group([&](uint32_t d) { lk_issue<2, MODE>(d, tm + LK_TA, b0); });
        group([&](uint32_t d) { lk_issue<1, MODE>(d, tm + LK_TA, b0); });
        group([&](uint32_t d) { lk_issue<0, MODE>(d, tm + LK_TA, b0); });
        if (ok && one) tc::mma_commit(&bar.done);
        __syncwarp();
      }
      // every MMA has ended before the tensor memory is released, no copy lands
      // after the block's end
      if (nkw > 0 && ok) wait(&bar.done, nk - 1);
      if (!ok && one) {
        *abort = 1;
        atomicExch(&err[b], 1);
        tc::mma_commit(&bar.drain);
        tc::mbar_wait(&bar.drain, 0u, 200000000LL);
      }
      __syncwarp();
      if (MODE == 0)
        for (int k = max(0, ncopy - 2); k < ncopy; ++k)
          tc::mbar_wait(&bar.b[k & 1], (uint32_t)((k >> 1) & 1), 200000000LL);
      if (warp > LK_CW) {
        // copies of chunk k into the staging buffers, zero outside the operands:
        // lane = row r (mode 1: the real parts, two rows r of 8 bytes per
        // 16-byte element)
        const zdf *A = p.A + b * p.sA;
        const zdf *Bm = p.Bm + b * p.sB;
        for (int k = 0; k < nk && ok; ++k) {
          if (k > 0) wait(&bar.st_free, k - 1);
          if (!ok) break;
          const int r0 = p.rbeg + CR * (kc_beg + k) + lane;
#pragma unroll 4
          for (int c = warp - LK_CW - 1; c < 128; c += LK_LW) {
            const zdf *src = A + p.lda * (c0 + c);
            if (MODE == 0) {
              const bool v = r0 < n && c0 + c < na;
              cp_async16(&stA[c * LK_LD + lane], v ? src + r0 : A, v);
            } else {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const bool v = r0 + 32 * h < n && c0 + c < na;
                cp_async8((df *)(stA + c * LK_LD) + lane + 32 * h, v ? src + r0 + 32 * h : A, v);
              }
            }
          }
          if (MODE == 1) {
#pragma unroll 4
            for (int jj = warp - LK_CW - 1; jj < 64; jj += LK_LW) {
              const int j = jj >> 1, rr = 32 * (jj & 1);
              const bool v = r0 + rr < n && j0 + j < nj;
              cp_async16(&stB[j * LK_LDB + lane + rr], v ? Bm + r0 + rr + p.ldb * (j0 + j) : Bm, v);
            }
          }
          tc::mbar_arrive_cp(&bar.st_full);
        }
        if (!ok && lane == 0) {
          *abort = 1;
          atomicExch(&err[b], 1);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");  // no copy may land after the block's end
      }
    } else {
      asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
      df acc[16];  // re and im of this thread's 8 columns
#pragma unroll
      for (int k = 0; k < 16; ++k) acc[k] = df{0.f, 0.f};
      auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * LK_CW) : "memory"); };
      Fixed56 f[16];  // K = 16 ks ... of row cl
      int En = 0;     // and the row's exponent
      int eb = 0;     // mode 1: exponent of column lane
      // the integers of chunk k from the staging buffers (mode 1: also B's
      // slices of it), which then take chunk k + 1
      auto prep = [&](int k) {
        ok = __all_sync(0xffffffffu, ok && wait_phase(&bar.st_full, (uint32_t)(k & 1), abort));
        df x[16];
        if (MODE == 0) {
#pragma unroll
          for (int t = 0; t < 16; ++t) x[t] = ((const df *)&stA[cl * LK_LD + 16 * (ks & 1) + t])[ks >> 1];
        } else {
#pragma unroll
          for (int t = 0; t < 16; t += 2) {
            const zdf two = stA[cl * LK_LD + 8 * ks + t / 2];
            x[t] = two.re;
            x[t + 1] = two.im;
          }
        }
        float amax = 0.f;
#pragma unroll
        for (int t = 0; t < 16; ++t) amax = max_abs(amax, x[t].hi);
        float *row = sRow[k & 1], *col = sCol[k & 1];
        row[ks * 128 + cl] = amax;
        df yr[4], yi[4];  // mode 1: B column lane, rows r = 4 warp ... of the chunk
        if (MODE == 1) {
          float bmax = 0.f;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const zdf y = stB[lane * LK_LDB + 4 * warp + t];
            yr[t] = y.re;
            yi[t] = y.im;
            bmax = max_abs(max_abs(bmax, y.re.hi), y.im.hi);
          }
          col[warp * 32 + lane] = bmax;
        }
        sync();  // the maxima are there (two sets: the next chunk's may come while these are read)
        if (lane == 0) tc::mbar_arrive(&bar.st_free);
        if (MODE == 1) {
          float bmax = 0.f;
#pragma unroll
          for (int q = 0; q < 16; ++q) bmax = max_abs(bmax, col[q * 32 + lane]);
          const int E = grid_exp(bmax);
          Fixed56 fr[4], fi[4];
          to_fixed<4>(yr, E, false, fr);
          to_fixed<4>(yi, E, true, fi);
          uint8_t *dst = sBop + (k & 1) * BOP + (warp >> 2) * 1024 + tc::core_off(lane, 4 * (warp & 3));
          auto put = [&](auto dig, int s) {
            *(uint2 *)(dst + s * TC_KS * 1024) = make_uint2(dig(fr[0], fr[1]), dig(fr[2], fr[3]));
            *(uint2 *)(dst + (TC_S + s) * TC_KS * 1024) = make_uint2(dig(fi[0], fi[1]), dig(fi[2], fi[3]));
          };
          put([](Fixed56 a, Fixed56 c) { return digit2<0>(a, c); }, 0);
          put([](Fixed56 a, Fixed56 c) { return digit2<1>(a, c); }, 1);
          put([](Fixed56 a, Fixed56 c) { return digit2<2>(a, c); }, 2);
          put([](Fixed56 a, Fixed56 c) { return digit2<3>(a, c); }, 3);
          put([](Fixed56 a, Fixed56 c) { return digit2<4>(a, c); }, 4);
          put([](Fixed56 a, Fixed56 c) { return digit2<5>(a, c); }, 5);
          put([](Fixed56 a, Fixed56 c) { return digit2<6>(a, c); }, 6);
          eb = E;  // of column lane
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        En = grid_exp(max_abs(max_abs(row[cl], row[128 + cl]), max_abs(row[256 + cl], row[384 + cl])));
        to_fixed<16>(x, En, false, f);
      };
      const uint32_t lane_base = tm + ((uint32_t)(32 * lg) << 16);
      auto store = [&](auto dig, int s) {
        uint32_t w[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) w[t] = dig(f[2 * t], f[2 * t + 1]);
        tc::tmem_st8(lane_base + LK_TA + (s * TC_KS + ks) * 8, w);
      };
      auto ready = [&] {
        tc::tmem_st_wait();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bar.a_ready);
      };
      prep(0);
      store([](Fixed56 a, Fixed56 c) { return digit2<6>(a, c); }, 6);
      store([](Fixed56 a, Fixed56 c) { return digit2<5>(a, c); }, 5);
      store([](Fixed56 a, Fixed56 c) { return digit2<4>(a, c); }, 4);
      store([](Fixed56 a, Fixed56 c) { return digit2<3>(a, c); }, 3);
      store([](Fixed56 a, Fixed56 c) { return digit2<2>(a, c); }, 2);
      store([](Fixed56 a, Fixed56 c) { return digit2<1>(a, c); }, 1);
      store([](Fixed56 a, Fixed56 c) { return digit2<0>(a, c); }, 0);
      ready();
      for (int k = 0; k < nk; ++k) {
        const int Ec = En;
        const int ebc = MODE ? eb : p.Ex[b * p.sEx + 32 * (kc_beg + k) + lane];  // of column lane
        const bool more = k + 1 < nk;
        if (more) prep(k + 1);
        df s[16];
        int g = k * TC_S;
        auto stage = [&](auto fold, auto dig, int u) {
          const int slot = g & (LK_ACC - 1);
          ok = __all_sync(0xffffffffu, ok && wait_phase(&bar.acc[slot], (uint32_t)((g / LK_ACC) & 1), abort));
          tc::fence_after();
          float a[16];
          tc::tmem_ld8(lane_base + slot * 64 + 8 * ks, a);
          tc::tmem_ld8(lane_base + slot * 64 + 32 + 8 * ks, a + 8);
          tc::tmem_ld_wait();
#pragma unroll
          for (int t = 0; t < 16; ++t) fold(s[t], a[t]);
          if (more) store(dig, u);
          tc::fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&bar.acc_free[slot]);
          ++g;
        };
        stage([](df &v, float a) { fold_up<6>(v, a); }, [](Fixed56 a, Fixed56 c) { return digit2<6>(a, c); }, 6);
        stage([](df &v, float a) { fold_up<5>(v, a); }, [](Fixed56 a, Fixed56 c) { return digit2<5>(a, c); }, 5);
        stage([](df &v, float a) { fold_up<4>(v, a); }, [](Fixed56 a, Fixed56 c) { return digit2<4>(a, c); }, 4);
        stage([](df &v, float a) { fold_up<3>(v, a); }, [](Fixed56 a, Fixed56 c) { return digit2<3>(a, c); }, 3);
        stage([](df &v, float a) { fold_up<2>(v, a); }, [](Fixed56 a, Fixed56 c) { return digit2<2>(a, c); }, 2);
        stage([](df &v, float a) { fold_up<1>(v, a); }, [](Fixed56 a, Fixed56 c) { return digit2<1>(a, c); }, 1);
        stage([](df &v, float a) { fold_up<0>(v, a); }, [](Fixed56 a, Fixed56 c) { return digit2<0>(a, c); }, 0);
        if (more) ready();
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const float sc = pow2f(Ec + __shfl_sync(0xffffffffu, ebc, 8 * ks + t) - 16);
          acc[t] = df_add(acc[t], df{__fmul_rn(s[t].hi, sc), __fmul_rn(s[t].lo, sc)});
          acc[8 + t] = df_add(acc[8 + t], df{__fmul_rn(s[8 + t].hi, sc), __fmul_rn(s[8 + t].lo, sc)});
        }
      }
      if (!ok && lane == 0) {
        *abort = 1;
        atomicExch(&err[b], 1);
      }
      write(acc);
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == LK_CW) tc::tmem_dealloc(tm, 512);
  } else if (warp < LK_CW) {
    df zero[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) zero[k] = df{0.f, 0.f};
    write(zero);
  }
}

}  // namespace

// PARPHOM_GPU_TC=0 selects the CUDA-core trailing update in the double-float
// form (both are the library's own kernels; the tensor-core one is default).
bool tc_enabled() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("PARPHOM_GPU_TC");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

size_t her2k_tc_bytes(int64_t nmax) { return (size_t)((nmax + 127) / 128) * TC_RBLK; }
int64_t her2k_tc_exps(int64_t nmax) { return 2 * ((nmax + 127) / 128) * 128; }

// Opt the tensor-core kernels into their shared memory on the current device
// (the attribute is per device; done once per device, outside any capture).
cudaError_t prepare_her2k_tc() {
  static std::mutex mu;
  static bool done[PP_MAX_DEVICES] = {};
  const int dev = device_index();
  std::lock_guard<std::mutex> g(mu);
  if (dev >= 0 && done[dev]) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_cupd_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, CU_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_longk_tc<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, lk_smem<0>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_longk_tc<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, lk_smem<1>());
  if (e == cudaSuccess && dev >= 0) done[dev] = true;
  return e;
}

namespace {
cudaError_t launch_slices(const TcSliceSrc &src, int rows_max, EigWork &w, int k0, int jb, uint8_t *S, int64_t blk,
                          int *E, int es, int eo, cudaStream_t s) {
  const int rows = (rows_max + 127) / 128 * 128;
  if (rows <= 0) return cudaSuccess;
  PP_KT(KT_HER2K, s, (k_tc_slices<<<dim3(rows / 4, w.B), 128, 0, s>>>(src, w.nvec, k0, jb, S, w.sTcS, blk, E, w.sTcE,
                                                                      es, eo)));
  count_launch(1);
  return cudaGetLastError();
}
}  // namespace

// One-shot stall of the test hook: the global batch index of the matrix
// and the wait's limit in SM clocks (-1: not armed).
static std::mutex g_stall_mu;
static int64_t g_stall_matrix = -1;
static long long g_stall_cycles = 0;

void arm_tc_stall(int64_t matrix, long long cycles) {
  std::lock_guard<std::mutex> g(g_stall_mu);
  g_stall_matrix = matrix;
  g_stall_cycles = cycles;
}
bool tc_stall_armed() {
  std::lock_guard<std::mutex> g(g_stall_mu);
  return g_stall_matrix >= 0;
}
// The stall for a launch over batch matrices [boff, boff + B): consumed by
// the first launch that covers the armed matrix.
static int take_stall(const EigWork &w, long long *cycles) {
  std::lock_guard<std::mutex> g(g_stall_mu);
  if (g_stall_matrix < w.boff || g_stall_matrix >= (int64_t)w.boff + w.B) return -1;
  const int b = (int)(g_stall_matrix - w.boff);
  *cycles = g_stall_cycles;
  g_stall_matrix = -1;
  return b;
}

// Column blocks per CTA for `tiles` tiles of 128 x 64 per matrix: up to 4 (the
// 112 KB row operand is fetched once per CTA and product), fewer while that
// leaves SMs without a CTA.
static int cu_blocks(int64_t tiles, int B) {
  int k = 4;
  while (k > 1 && tiles * B < (int64_t)k * device_sms()) k /= 2;
  return k;
}

// A(k1:n, k1:n) -= V W^H + W V^H, lower triangle (panel k0 of width jb).
cudaError_t her2k_tc(EigWork &w, int k0, int jb, cudaStream_t s) {
  const int k1 = k0 + jb;
  const int mmax = w.nmax - k1;
  if (mmax <= 0) return cudaSuccess;
  const int64_t sW = (int64_t)w.lda * w.nb;
  const zdf *A = (const zdf *)w.A;
  // V rows (block part 0) and W rows (block part 1) of the trailing block
  PP_CUDA_TRY(launch_slices(TcSliceSrc{A + w.lda * k0, w.sA, 1, w.lda, k1, 0, 1, 0}, mmax, w, k0, jb, w.tcS,
                            TC_RBLK, w.tcE, 2, 0, s));
  PP_CUDA_TRY(launch_slices(TcSliceSrc{(const zdf *)w.W, sW, 1, w.lda, k1, 0, 0, 0}, mmax, w, k0, jb,
                            w.tcS + TC_OP, TC_RBLK, w.tcE, 2, 1, s));
  TcUpdate u{};
  u.C = (zdf *)w.A;
  u.ldc = w.lda;
  u.sC = w.sA;
  u.rbase = u.cbase = k1;
  u.ncols_fixed = 0;
  u.tri = 1;
  u.nprod = 2;
  const TcOperand V{w.tcS, w.sTcS, TC_RBLK, w.tcE, w.sTcE, 2, 0};
  const TcOperand Wo{w.tcS + TC_OP, w.sTcS, TC_RBLK, w.tcE, w.sTcE, 2, 1};
  u.x[0] = V;
  u.y[0] = Wo;
  u.x[1] = Wo;
  u.y[1] = V;
  u.stall_b = take_stall(w, &u.stall_cycles);
  const int nrb = (mmax + 127) / 128;
  u.cbs = cu_blocks(nrb * (nrb + 1) / 2 * (128 / CU_N), w.B);
  const int nq = (128 / CU_N * nrb + u.cbs - 1) / u.cbs;
  PP_KT(KT_HER2K, s, (k_cupd_tc<<<dim3(nq, nrb, w.B), CU_NT, CU_SMEM, s>>>(u, w.nvec, w.tcErr)));
  count_launch(1);
  return cudaGetLastError();
}

// X(k0+1:n, 0:ncols) -= V Y with V the Householder vectors of panel k0 (width
// jb) and Y (jb x ncols) at Yb[a ldy + c]: the update of the compact-WY
// back-transform as X Y'^H with Y'(c, a) = conj(Y(a, c)).
cudaError_t applyV_tc(EigWork &w, int k0, int jb, zdf *X, int64_t ldx, int64_t sX, const zdf *Yb, int64_t ldy,
                      int64_t sY, int ncols, cudaStream_t s) {
  const int r1 = k0 + 1;
  const int mmax = w.nmax - r1;
  if (mmax <= 0 || ncols <= 0) return cudaSuccess;
  const zdf *A = (const zdf *)w.A;
  const int64_t vbl = (int64_t)((w.nmax + 127) / 128) * TC_OP;  // the Y' slices follow the V slices
  const int64_t yexp = (w.nmax + 127) / 128 * 128;
  PP_CUDA_TRY(launch_slices(TcSliceSrc{A + w.lda * k0, w.sA, 1, w.lda, r1, 0, 1, 0}, mmax, w, k0, jb, w.tcS, TC_OP,
                            w.tcE, 1, 0, s));
  PP_CUDA_TRY(launch_slices(TcSliceSrc{Yb, sY, 1, ldy, 0, ncols, 0, 1}, ncols, w, k0, jb, w.tcS + vbl, TC_OP,
                            w.tcE + yexp, 1, 0, s));
  TcUpdate u{};
  u.C = X;
  u.ldc = ldx;
  u.sC = sX;
  u.rbase = r1;
  u.cbase = 0;
  u.ncols_fixed = ncols;
  u.tri = 0;
  u.nprod = 1;
  u.stall_b = -1;
  u.x[0] = TcOperand{w.tcS, w.sTcS, TC_OP, w.tcE, w.sTcE, 1, 0};
  u.y[0] = TcOperand{w.tcS + vbl, w.sTcS, TC_OP, w.tcE + yexp, w.sTcE, 1, 0};
  u.x[1] = u.x[0];
  u.y[1] = u.y[0];
  const int nrb = (mmax + 127) / 128, ncb = (ncols + CU_N - 1) / CU_N;
  u.cbs = cu_blocks(nrb * ncb, w.B);
  const int nq = (ncb + u.cbs - 1) / u.cbs;
  PP_KT(KT_APPLYV, s, (k_cupd_tc<<<dim3(nq, nrb, w.B), CU_NT, CU_SMEM, s>>>(u, w.nvec, w.tcErr)));
  count_launch(1);
  return cudaGetLastError();
}

// Wp(a, c) = (V^H X)(a, c) over the rows r > k0 (V: panel k0 of width jb),
// c < ncols; the rows in vhx_tc_splits(w) ranges, a split-K slot of Wp each.
int vhx_tc_splits(const EigWork &w) { return std::max(1, std::min(4, w.ksplit)); }

cudaError_t vhx_tc(EigWork &w, int k0, int jb, const zdf *X, int64_t ldx, int64_t sX, int ncols, zdf *Wp,
                   int64_t ldwp, int64_t sWp, cudaStream_t s) {
  if (ncols <= 0) return cudaSuccess;
  LongK p{};
  p.A = X;
  p.lda = ldx;
  p.sA = sX;
  p.Bm = (const zdf *)w.A + w.lda * k0;
  p.ldb = w.lda;
  p.sB = w.sA;
  p.k0 = k0;
  p.jb = jb;
  p.rbeg = k0 + 1;
  p.ncols_a = ncols;
  p.out = Wp;
  p.ldo = ldwp;
  p.sO = sWp;
  // the slices of the panel and their exponents: the scratch that the update X -= V Y takes after this
  p.S = w.tcS;
  p.sS = w.sTcS;
  p.Ex = w.tcE;
  p.sEx = w.sTcE;
  const int nck = (w.nmax - p.rbeg + 31) / 32;
  if (nck > 0) {
    PP_KT(KT_VHX, s, (k_longk_bslice<<<dim3(nck, w.B), 128, 0, s>>>(p, w.nvec, w.tcS, w.tcE)));
    count_launch(1);
  }
  PP_KT(KT_VHX, s, (k_longk_tc<0><<<dim3((ncols + 127) / 128, vhx_tc_splits(w), w.B), LK_NT, lk_smem<0>(), s>>>(
                       p, w.nvec, w.tcErr)));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t xhz_tc(EigWork &w, const zdf *X, int64_t ldx, int64_t sX, int nrows, const zdf *Z, int64_t ldz,
                   int64_t sZ, zdf *Eb, int64_t lde, int64_t sE, cudaStream_t s) {
  if (nrows <= 0) return cudaSuccess;
  LongK p{};
  p.A = Z;
  p.lda = ldz;
  p.sA = sZ;
  p.Bm = X;
  p.ldb = ldx;
  p.sB = sX;
  p.nrows_b = nrows;
  p.rbeg = 0;
  p.rng = w.rng;
  p.out = Eb;
  p.ldo = lde;
  p.sO = sE;
  PP_KT(KT_XHZ, s, (k_longk_tc<1><<<dim3((nrows + 31) / 32, (w.mcap + 127) / 128, w.B), LK_NT, lk_smem<1>(), s>>>(
                       p, w.nvec, w.tcErr)));
  count_launch(1);
  return cudaGetLastError();
}

}  // namespace pp
