// Batched Hermitian eigensolver with pzheevx semantics (range A/I/V, abstol,
// optional eigenvectors) for the phonon hot path.
//
// Stages (each a set of batched kernels; matrix b of the batch is picked by
// blockIdx.y/z and may have its own order nvec[b]):
//  1. Householder reduction to real symmetric tridiagonal form, lower
//     formulation, blocked in panels of nb columns: the per-column work
//     (column update, reflector, Hermitian matrix-vector product and its
//     panel corrections) follows the zlatrd recurrence; after each panel the
//     trailing matrix gets the rank-2nb update A -= V W^H + W V^H.  The full
//     Hermitian square is kept so that every matrix-vector pass reads
//     coalesced columns (only its lower triangle is read after assembly).
//     A = Q T Q^H with Q = H(0) H(1) ... H(n-2), H(i) = I - tau_i v_i v_i^H.
//  2. Eigenvalues of T by Sturm-count bisection, one thread per eigenvalue
//     index, with the dstebz tolerance rule max(abstol, pivmin,
//     2 ulp max(|lo|,|hi|)): FP32 counts first, then FP64 ones (mixed form:
//     double-float ones, down to 4 x 2^-44 ||T||).
//  3. Eigenvectors of T by inverse iteration with partial-pivoting LU of
//     T - lambda I, one thread per eigenvalue cluster, modified Gram-Schmidt
//     inside clusters (consecutive eigenvalues closer than 1e-7 ||T||), then
//     a Gram-Schmidt pass over looser clusters (closer than 1e-5 ||T||).
//     Always FP64.
//  4. Back-transform E = Q Z, panel by panel from the last, with the compact
//     WY form I - V Tf V^H (zlarft forward/columnwise).
// Stages 1 and 4 are templated on the real arithmetic R: double (plain FP64
// form) or df (double-float on the FP32 pipes, the mixed form).
#include <atomic>
#include <algorithm>
#include <mutex>
#include <cfloat>
#include <type_traits>
#include <cstdio>
#include <cstdlib>

#include "pp_internal.cuh"
#include "pp_sums.cuh"

namespace pp {

template <class R>
using C = cx<R>;

static inline int cdiv(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }
__device__ __forceinline__ int cdiv_dev(int a, int b) { return (a + b - 1) / b; }

// ---------------------------------------------------------------------------
// block reductions (double / z64)
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int NT>
__device__ double block_sum(double v, double *sh) {
  v = warp_sum(v);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x < 32) {
    r = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  if (threadIdx.x == 0) sh[0] = r;
  __syncthreads();
  r = sh[0];
  __syncthreads();
  return r;
}
// ===========================================================================
// Stage 1: reduction to tridiagonal form
// ===========================================================================
constexpr int TR_NT = 256;   // threads of the column kernels

// The mat-vec and the column steps of a panel are launched as dependent
// launches: a kernel may start once every block of the one before has called
// dep_go, does what does not read that kernel's results, and waits in dep_wait
// until it has completed (every block waits, before any return, so that
// completion carries over the whole chain; dep_go comes after dep_wait, so that
// all earlier kernels but the one before have completed when a kernel starts).
// What is loaded before dep_wait may be what a completed kernel wrote to lines that
// this SM's L1 has held before, and no rule says that the early start clears it: those
// loads go past L1 (load_l2, cp.async.cg).  The mat-vec requests its first tile early,
// the column step its panel rows, v and the next column.  A pass: n = 1092 (FP64,
// eigenvalues) 38.6 -> 30.3 ms, n = 2604 with
// vectors 168 -> 156 ms, n = 1092 x 16 64.8 -> 61.1 ms.  dep_go is called late
// (a block's last tile, a column's last phase): blocks that wait early hold
// slots that other streams' kernels need (column step calling it first: 166 and
// 63.9 ms).
PP_D void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
PP_D void dep_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class R>
PP_D cx<R> load_l2(const cx<R> *p) {
  const float4 v = __ldcg((const float4 *)p);
  return *(const cx<R> *)&v;
}
template <class... P, class... A>
static cudaError_t launch_dep(void (*kernel)(P...), dim3 grid, int threads, size_t smem, int cluster, bool dep,
                              cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  cfg.attrs = at;
  if (cluster) {
    at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    at[cfg.numAttrs].val.clusterDim.x = cluster;
    at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (dep) {
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

template <class R>
__device__ __forceinline__ R shfl_xor_real(R x, int o) {
  R y;
  float *dst = (float *)&y;
  const float *p = (const float *)&x;
#pragma unroll
  for (int f = 0; f < (int)(sizeof(R) / sizeof(float)); ++f) dst[f] = __shfl_xor_sync(0xffffffffu, p[f], o);
  return y;
}

// Sums of y and of z over each group of 8 consecutive lanes, in every lane of
// the group.  Halving: after the first exchange half of the lanes carry y and
// half z, after the second one component each, so a lane makes 4 additions
// instead of the 12 of two plain butterflies (an FP64 addition holds the pipe
// for 16 cycles per warp).
template <class R>
__device__ __forceinline__ void group8_sum(C<R> &y, C<R> &z) {
  const int lane = threadIdx.x & 31;
  const bool hz = (lane & 4) != 0, him = (lane & 2) != 0;
  const C<R> keep = hz ? z : y, send = hz ? y : z;
  const C<R> got{shfl_xor_real(send.re, 4), shfl_xor_real(send.im, 4)};
  const C<R> m = cadd(keep, got);
  const R k1 = him ? m.im : m.re, s1 = him ? m.re : m.im;
  R v = RT<R>::add(k1, shfl_xor_real(s1, 2));
  v = RT<R>::add(v, shfl_xor_real(v, 1));
  const int g = lane & ~7;
  y = C<R>{shfl_real(v, g), shfl_real(v, g + 2)};
  z = C<R>{shfl_real(v, g + 4), shfl_real(v, g + 6)};
}

// ---- the reflector's scalars (zlarfg): from |x|^2 and alpha, beta =
// -copysign(sqrt(|alpha|^2 + |x|^2), Re alpha), tau = ((beta - Re alpha) /
// beta, -Im alpha / beta) and 1 / (alpha - beta).  All lanes of a warp take
// part; the four quotients run in lanes 0-3 (one division in time).
// A sum of x values scaled by 2^-e per value (squares by 2^-2e) keeps the
// double-float form clear of the float range.
template <class R>
struct Reflector {
  C<R> tau, scale;  // scale belongs to values multiplied by prescale()
  typename Sum<R>::T beta, t_re, t_im;
  int e;  // beta is to be multiplied by 2^e
  int skip;
};
__device__ __forceinline__ float pow2_clamped(int e) {  // 2^e, |e| <= 126
  return __int_as_float((e + 127) << 23);
}
__device__ __forceinline__ Reflector<double> reflector_scalars(double xn2, int, C<double> al) {
  Reflector<double> f;
  const int lane = threadIdx.x & 31;
  f.e = 0;
  f.skip = xn2 == 0.0 && al.im == 0.0;
  const double nrm = sqrt(al.re * al.re + al.im * al.im + xn2);
  f.beta = f.skip ? al.re : -copysign(nrm, al.re);
  const double dr = al.re - f.beta, di = al.im;
  const double num = lane == 0 ? -dr : (lane == 2 ? dr : -di);
  const double den = lane < 2 ? f.beta : dr * dr + di * di;
  const double quo = f.skip ? 0.0 : num / den;
  f.t_re = __shfl_sync(0xffffffffu, quo, 0);
  f.t_im = __shfl_sync(0xffffffffu, quo, 1);
  f.tau = C<double>{f.t_re, f.t_im};
  f.scale = C<double>{__shfl_sync(0xffffffffu, quo, 2), __shfl_sync(0xffffffffu, quo, 3)};
  return f;
}
__device__ __forceinline__ tf tf_norm(tf x) {
  float s, e, t, u;
  two_sum(x.a, x.b, s, e);
  two_sum(e, x.c, t, u);
  tf r;
  fast_two_sum(s, t, r.a, r.b);
  r.c = u;
  return r;
}
__device__ __forceinline__ tf tf_scale(tf x, float f) {  // f a power of two
  return tf{__fmul_rn(x.a, f), __fmul_rn(x.b, f), __fmul_rn(x.c, f)};
}
__device__ __forceinline__ tf tf_mulf(float q, tf x) {
  const float p = __fmul_rn(q, x.a), pe = __fmaf_rn(q, x.a, -p);
  const float r = __fmul_rn(q, x.b), re = __fmaf_rn(q, x.b, -r);
  float s, e;
  two_sum(pe, r, s, e);
  return tf{p, s, __fadd_rn(__fmaf_rn(q, x.c, re), e)};
}
// The same in expansions of three floats: square root and quotients from a
// float estimate and two exact-remainder corrections (Newton / long division),
// about 2^-66 relative -- more than the FP64 forms, at float latency.
__device__ __forceinline__ Reflector<df> reflector_scalars(tf xn2, int ex, C<df> al) {
  typedef Sum<df> S;
  Reflector<df> f;
  const int lane = threadIdx.x & 31;
  const int ea = (int)(__float_as_uint(fmaxf(fabsf(al.re.hi), fabsf(al.im.hi))) >> 23) - 127;
  const int E = max(ex, min(max(ea, -120), 120));
  const float fa = pow2_clamped(-E);
  const int d2 = 2 * (ex - E);
  const df ar{__fmul_rn(al.re.hi, fa), __fmul_rn(al.re.lo, fa)}, ai{__fmul_rn(al.im.hi, fa), __fmul_rn(al.im.lo, fa)};
  f.e = E;
  f.skip = xn2.a == 0.f && al.im.hi == 0.f;
  const tf s = tf_norm(S::add(tf_scale(xn2, d2 < -126 ? 0.f : pow2_clamped(d2)), S::add(S::mul(ar, ar), S::mul(ai, ai))));
  // sqrt
  const float y = rsqrtf(s.a), r = __fmul_rn(s.a, y), hy = 0.5f * y;
  const float p = __fmul_rn(r, r), pe = __fmaf_rn(r, r, -p);
  const float c1 = __fmul_rn(__fadd_rn(__fsub_rn(__fsub_rn(s.a, p), pe), s.b), hy);
  df h;
  fast_two_sum(r, c1, h.hi, h.lo);
  const tf rem = S::sub(s, S::mul(h, h));
  tf beta{h.hi, h.lo, __fmul_rn(__fadd_rn(rem.a, __fadd_rn(rem.b, rem.c)), hy)};
  if (!signbit(ar.hi)) beta = tf{-beta.a, -beta.b, -beta.c};
  if (f.skip) beta = S::from(ar);
  f.beta = beta;
  // quotients
  const tf dr = tf_norm(S::sub(S::from(ar), beta));  // alpha_r - beta: no cancellation
  const df dh{dr.a, dr.b};
  tf dd = S::mul(dh, dh);
  dd.c = __fmaf_rn(2.f * dr.a, dr.c, dd.c);
  const tf den = tf_norm(lane < 2 ? beta : S::add(dd, S::mul(ai, ai)));
  const tf num = lane == 0 ? tf{-dr.a, -dr.b, -dr.c} : (lane == 2 ? dr : tf{-ai.hi, -ai.lo, 0.f});
  const float rc = __frcp_rn(den.a);
  const float q0 = __fmul_rn(num.a, rc);
  const tf m1 = tf_norm(S::sub(num, tf_mulf(q0, den)));
  const float q1 = __fmul_rn(m1.a, rc);
  const tf m2 = tf_norm(S::sub(m1, tf_mulf(q1, den)));
  tf q = tf_norm(tf{q0, q1, __fmul_rn(m2.a, rc)});
  if (f.skip) q = S::zero();
  const df qd = S::toR(q);
  f.tau = C<df>{shfl_real(qd, 0), shfl_real(qd, 1)};
  f.scale = C<df>{shfl_real(qd, 2), shfl_real(qd, 3)};
  f.t_re = tf{__shfl_sync(0xffffffffu, q.a, 0), __shfl_sync(0xffffffffu, q.b, 0), __shfl_sync(0xffffffffu, q.c, 0)};
  f.t_im = tf{__shfl_sync(0xffffffffu, q.a, 1), __shfl_sync(0xffffffffu, q.b, 1), __shfl_sync(0xffffffffu, q.c, 1)};
  return f;
}
__device__ __forceinline__ C<double> prescale(C<double> x, int) { return x; }
__device__ __forceinline__ C<df> prescale(C<df> x, int e) {
  const float f = pow2_clamped(-e);
  return C<df>{df{__fmul_rn(x.re.hi, f), __fmul_rn(x.re.lo, f)}, df{__fmul_rn(x.im.hi, f), __fmul_rn(x.im.lo, f)}};
}
__device__ __forceinline__ float magnitude(C<double>) { return 0.f; }
__device__ __forceinline__ float magnitude(C<df> x) { return fmaxf(fabsf(x.re.hi), fabsf(x.im.hi)); }

// ---- the mat-vec of the FP64 form
// Lower-triangle Hermitian mat-vec y = A v on the trailing block [i+1, n),
// over the lower tile pairs (R >= C) of HL_T x HL_T: a tile is read once and
// gives both A_RC v_C (into slot C of the rows of R) and A_RC^H v_R (into
// slot R of the rows of C).  Every row receives exactly one partial per slot
// 0 .. ntiles-1, summed by the column step (k_wpart, k_colstep).  Blocks are
// persistent over a strided set of tile pairs with two shared-memory buffers: the
// next tile (and its two vector pieces) is copied by cp.async while the FP64
// arithmetic of the current one runs.
constexpr int HL_T = 32;         // tile of large trailing blocks
constexpr int HL_TS = 16;        // tile of trailing blocks up to HL_SMALL rows: four times the tiles, so that
constexpr int HL_SMALL = 128;    // more SMs' FP64 pipes take part (n = 84: 9.1 -> 7.9 us between events)
constexpr int HL_BPS = 6;        // resident blocks per SM
constexpr int HL_UNROLL = 4;     // inner-loop unrolling (keeps the kernel's code small)
__host__ __device__ __forceinline__ int hl_tile(int rows) { return rows <= HL_SMALL ? HL_TS : HL_T; }
__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void tile_pair(int p, int &Rt, int &Ct) {
  Rt = (int)((sqrtf(8.0f * (float)p + 1.0f) - 1.0f) * 0.5f);
  while ((Rt + 1) * (Rt + 2) / 2 <= p) ++Rt;
  while (Rt * (Rt + 1) / 2 > p) --Rt;
  Ct = p - Rt * (Rt + 1) / 2;
}
// One of the panel products of column i, by 128 threads (t) of one block of
// the double-float mat-vec's launch: X[c] = V(:,c)^H v (c < jj), X[jj+c] =
// W(:,c)^H v over rows [i+1, n).  They need only v, so they run beside the mat-vec instead of in a launch of
// their own.  Each thread adds up 4 rows at a time, the blocks of 4 in three floats.
__device__ __forceinline__ void panel_dot(const zdf *A, const zdf *W, int64_t lda, int n, int i, int k0, int jj,
                                          int c2, int t, Sum<df>::T (*red)[4], zdf *X) {
  typedef Sum<df> S;
  typedef S::T T;
  constexpr int NT = 128;
  const bool some = c2 < 2 * jj;  // (the last block's spare groups only pass the barrier)
  const bool useW = c2 >= jj;
  const int c = useW ? c2 - jj : c2;
  const zdf *Xc = useW ? (W + lda * c) : (A + lda * (k0 + c));
  const zdf *v = A + lda * i;
  T sr = S::zero(), si = S::zero();
  auto flush = [&](zdf acc) {
    acc = cfin(acc);
    sr = S::add(sr, S::from(acc.re));
    si = S::add(si, S::from(acc.im));
  };
  int r = some ? i + 1 + t : n;
  for (; r + 3 * NT < n; r += 4 * NT) {
    zdf x[4], y[4], acc = cz<df>();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x[u] = Xc[r + u * NT];
      y[u] = v[r + u * NT];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) cmacc(acc, x[u], y[u]);
    flush(acc);
  }
  zdf last = cz<df>();
  for (; r < n; r += NT) cmacc(last, Xc[r], v[r]);
  flush(last);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sr = S::add(sr, S::shfl_xor(sr, o));
    si = S::add(si, S::shfl_xor(si, o));
  }
  if ((t & 31) == 0) {
    red[0][t >> 5] = sr;
    red[1][t >> 5] = si;
  }
  __syncthreads();
  if (t == 0 && some) {
#pragma unroll
    for (int k = 1; k < NT / 32; ++k) {
      sr = S::add(sr, red[0][k]);
      si = S::add(si, red[1][k]);
    }
    X[c2] = zdf{S::toR(sr), S::toR(si)};
  }
}

// The same in FP64, one product per warp: a warp's sum takes 10 additions
// across lanes, a block's 40 and a barrier, and an FP64 addition holds the pipe
// for 16 cycles.
__device__ __forceinline__ void panel_dot_warp(const z64 *A, const z64 *W, int64_t lda, int n, int i, int k0, int jj,
                                               int c2, z64 *X) {
  if (c2 >= 2 * jj) return;
  const int lane = threadIdx.x & 31;
  const z64 *Xc = c2 >= jj ? W + lda * (c2 - jj) : A + lda * (k0 + c2);
  const z64 *v = A + lda * i;
  z64 acc{0.0, 0.0};
  int r = i + 1 + lane;
  for (; r + 3 * 32 < n; r += 4 * 32) {
    z64 x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x[u] = Xc[r + u * 32];
      y[u] = v[r + u * 32];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) cmacc(acc, x[u], y[u]);
  }
  for (; r < n; r += 32) cmacc(acc, Xc[r], v[r]);
  acc.re = warp_sum(acc.re);
  acc.im = warp_sum(acc.im);
  if (lane == 0) X[c2] = acc;
}

// blocks of the panel products: a warp each
__host__ __device__ __forceinline__ int hl_dots(int jj, int tile) { return (2 * jj + tile / 8 - 1) / (tile / 8); }
template <int HL_T>
__global__ void __launch_bounds__(4 * HL_T, HL_BPS * 32 / HL_T) k_hemv_lower(const z64 *Ab, int64_t lda, int64_t sA,
                                                              const int *nvec, int i, z64 *Pb, int64_t sP,
                                                              int64_t ldp, const z64 *Wb, int64_t sW, int k0,
                                                              int jj, z64 *X, int ldx) {
  constexpr int HL_LD = HL_T + 1;  // padded column stride of the shared tile
  constexpr int HL_NT = 4 * HL_T;
  __shared__ __align__(16) z64 tile[2][HL_T * HL_LD];  // tile[buf][c * HL_LD + r]
  __shared__ __align__(16) z64 vR[2][HL_T], vC[2][HL_T];
  __shared__ z64 red[2][2][HL_T];
  const int b = blockIdx.z;
  const int n = nvec[b];
  const int r0 = i + 1;
  const int nd = hl_dots(jj, HL_T);
  if (r0 >= n || hl_tile(n - r0) != HL_T || (int)blockIdx.x < nd) {
    dep_wait();
    dep_go();
    if (r0 >= n || hl_tile(n - r0) != HL_T) return;
    panel_dot_warp(Ab + b * sA, Wb + b * sW, lda, n, i, k0, jj, blockIdx.x * (HL_NT / 32) + threadIdx.x / 32, X + b * ldx);
    return;
  }
  const int bx = blockIdx.x - nd, gx = gridDim.x - nd;  // among the mat-vec's blocks
  const int nt = (n - r0 + HL_T - 1) / HL_T;
  const int npairs = nt * (nt + 1) / 2;
  if (bx >= npairs) {
    dep_wait();
    return;
  }
  const z64 *A = Ab + b * sA;
  const int tid = threadIdx.x;
  // copies of tile pair p into buffer buf (zero outside the matrix); the first
  // tile's before the column step has completed, which writes v only
  auto issue = [&](int p, int buf, bool first = false) {
    int Rt, Ct;
    tile_pair(p, Rt, Ct);
    const int rt0 = r0 + Rt * HL_T, ct0 = r0 + Ct * HL_T;
    // element (r, c) = (tid % HL_T, tid / HL_T + CS j), j < HL_T / CS
    constexpr int CS = HL_NT / HL_T;
    const int r = tid % HL_T, cb = tid / HL_T;
    const int rr = rt0 + r;
    const z64 *src = A + rr + lda * (ct0 + cb);
    z64 *dst = &tile[buf][cb * HL_LD + r];
#pragma unroll
    for (int j = 0; j < HL_T / CS; ++j) {
      const bool ok = rr < n && ct0 + cb + CS * j < n;
      cp_async16(dst + CS * j * HL_LD, ok ? (const void *)(src + CS * j * lda) : (const void *)A, ok);
    }
    if (first) dep_wait();
    if (tid < HL_T) {
      const int rr = rt0 + tid;
      cp_async16(&vR[buf][tid], rr < n ? (const void *)&A[rr + lda * i] : (const void *)A, rr < n);
    } else if (tid < 2 * HL_T) {
      const int cc = ct0 + tid - HL_T;
      cp_async16(&vC[buf][tid - HL_T], cc < n ? (const void *)&A[cc + lda * i] : (const void *)A, cc < n);
    }
    cp_async_commit();
  };
  // warps 0-1: A_RC v_C (thread = row, half of the columns each);
  // warps 2-3: A_RC^H v_R (thread = column, half of the rows each)
  const int lane = tid & (HL_T - 1), wid = tid / HL_T;
  const int prod = wid >> 1, half = wid & 1;
  constexpr int SPAN = HL_T / 2;
  issue(bx, 0, true);
  int buf = 0;
  for (int p = bx; p < npairs; p += gx) {
    if (p + gx < npairs) {
      issue(p + gx, buf ^ 1);
    } else {
      dep_go();
      cp_async_commit();  // an empty group keeps "all but the newest" meaning this tile
    }
    cp_async_wait1();
    __syncthreads();
    int Rt, Ct;
    tile_pair(p, Rt, Ct);
    const int rt0 = r0 + Rt * HL_T, ct0 = r0 + Ct * HL_T;
    const bool diag = (Rt == Ct);
    const z64 *tl = tile[buf];
    if (prod == 0) {
      z64 acc = z64{0.0, 0.0};
      const int r = lane;
      if (!diag) {
#pragma unroll HL_UNROLL
        for (int c = half * SPAN; c < half * SPAN + SPAN; ++c) cmac(acc, tl[c * HL_LD + r], vC[buf][c]);
      } else {  // diagonal tile: the upper part is the conjugate of the mirrored element
#pragma unroll HL_UNROLL
        for (int c = half * SPAN; c < half * SPAN + SPAN; ++c) {
          const z64 a = (r >= c) ? tl[c * HL_LD + r] : cconj(tl[r * HL_LD + c]);
          cmac(acc, a, vC[buf][c]);
        }
      }
      red[0][half][r] = cfin(acc);
    } else if (!diag) {
      z64 acc = z64{0.0, 0.0};
      const int c = lane;
#pragma unroll HL_UNROLL
      for (int r = half * SPAN; r < half * SPAN + SPAN; ++r) cmacc(acc, tl[c * HL_LD + r], vR[buf][r]);
      red[1][half][c] = cfin(acc);
    }
    __syncthreads();
    if (wid == 0 && rt0 + lane < n)
      Pb[b * sP + (int64_t)Ct * ldp + rt0 + lane] = cadd(red[0][0][lane], red[0][1][lane]);
    if (wid == 2 && !diag && ct0 + lane < n)
      Pb[b * sP + (int64_t)Rt * ldp + ct0 + lane] = cadd(red[1][0][lane], red[1][1][lane]);
    __syncthreads();  // the buffer and red are free for the next iteration
    buf ^= 1;
  }
  cp_async_wait0();
}

// ---- the mat-vec of the double-float form
// Lower-triangle Hermitian mat-vec on tiles of 64 rows x 32 columns of the
// trailing block.  Warps 0-3 form A_RC v_C (16 rows each; a lane: one row,
// half of the columns), warps 4-7 A_RC^H v_R (8 columns each; a lane: one
// column, 16 rows): every sum ends inside one warp, so that the only barrier
// per tile is the one that hands over its buffer.  In the two tiles on the
// diagonal the entries above it are masked in both products and the diagonal
// itself in the second.  Each CTA walks a run of consecutive tiles of the
// row-major tile list and keeps the row sums in registers along a tile row,
// so a row gets one partial per run that crosses its tile row and one per
// tile row from its own on (hv_slots) instead of one per 32 columns.  The
// runs depend on the order of the trailing block, the column of the panel and
// the number of SMs only.  The first CTAs of the grid form the panel products
// (panel_dot), 2 per CTA.
// A lane's 16 products of a tile are summed on their own (df_block) and added to
// the row's sum.
// Bound by instruction issue: 80 double-float lane operations per stored
// element (two complex multiply-adds of ten operations each), about 110 instructions
// in all where the 32 x 32 tiles of the earlier kernel took 152.  One matrix of order
// 4764, first columns: 66.5 us -> 53.5 us (3.4 TB/s), with twelve operations; all columns
// of 8 such matrices, the average: 139 us with twelve operations, 131 us with ten in
// two sums per tile (127 us with one sum along the row, whose rounding errors are
// larger than those of the twelve).
// Measured and not kept: packed f32x2 arithmetic (30% fewer instructions, but three
// shared-memory reads per vector entry: 57 us); bulk copies by a fetching warp
// with mbarriers (61 us: 1 KB copies are issued too slowly); tiles of 64 x 64.
constexpr int HV_R = 64, HV_C = 32, HV_LD = HV_R + 1;
constexpr int HV_NT = 256;
constexpr int HV_BPS = 3;  // resident CTAs per SM
constexpr int HV_TILE = HV_C * HV_LD * 16;
constexpr int HV_SMEM = 2 * HV_TILE + 2 * (HV_R + HV_C) * 16;
// CTAs of the panel products, CTAs left for the runs, tiles per run
__host__ __device__ __forceinline__ int hv_dots(int jj) { return jj; }
__host__ __device__ __forceinline__ int hv_ctas(int jj, int sms) {
  return HV_BPS * sms - hv_dots(jj) > 1 ? HV_BPS * sms - hv_dots(jj) : 1;
}
__host__ __device__ __forceinline__ int hv_run(int rows, int jj, int sms) {
  const int nt = (rows + HV_R - 1) / HV_R, tiles = nt * (nt + 1), g = hv_ctas(jj, sms);
  return (tiles + g - 1) / g;
}
// Partial slots of a row in tile row R of nt: runs first .. first + nseg - 1
// cross it (slots 0 .. nseg-1), tile rows R .. nt-1 hold its column (slots
// 2 nt + R .. 3 nt - 1).
__device__ __forceinline__ void hv_slots(int R, int run, int &first, int &nseg) {
  const int s = R * (R + 1);
  first = s / run;
  nseg = (s + 2 * R + 1) / run - first + 1;
}

__global__ void __launch_bounds__(HV_NT, HV_BPS) k_hemv_df(const zdf *Ab, int64_t lda, int64_t sA, const int *nvec,
                                                           int i, zdf *Pb, int64_t sP, int64_t ldp, const zdf *Wb,
                                                           int64_t sW, int k0, int jj, zdf *X, int ldx, int sms) {
  extern __shared__ __align__(16) unsigned char hv_smem[];
  zdf *tiles = (zdf *)hv_smem;              // [2][32 columns][HV_LD]
  zdf *vecs = tiles + 2 * HV_C * HV_LD;     // [2][v_R 64, v_C 32]
  const int b = blockIdx.y;
  const int n = nvec[b];
  const int r0 = i + 1;
  const zdf *A = Ab + b * sA;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nd = hv_dots(jj);
  if (r0 >= n || (int)blockIdx.x < nd) {
    dep_wait();
    dep_go();
    if (r0 >= n) return;
    const int g = warp >> 2;
    panel_dot(A, Wb + b * sW, lda, n, i, k0, jj, blockIdx.x * 2 + g, tid & 127,
                  (Sum<df>::T(*)[4])hv_smem + 2 * g,
                  X + b * ldx);
    return;
  }
  const int nt = (n - r0 + HV_R - 1) / HV_R;
  const int run = hv_run(n - r0, jj, sms);
  const int x = blockIdx.x - nd;
  int t = x * run;
  const int tend = min(t + run, nt * (nt + 1));
  if (t >= tend) {
    dep_wait();
    return;
  }
  int R = (int)((sqrtf(4.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while ((R + 1) * (R + 2) <= t) ++R;
  while (R * (R + 1) > t) --R;
  int Cc = t - R * (R + 1);
  int Ri = R, Ci = Cc, ti = t;  // the next tile to request
  // this thread's part of a tile: row tr, columns tc, tc + 4, ...
  const int tr = tid & (HV_R - 1), tc = tid / HV_R;
  // copies of the next tile and its vector pieces into buffer buf (zero
  // outside the matrix); an empty group past the run's end.  The first tile is
  // requested before the column step has completed, which writes v only.
  auto issue = [&](int buf, bool first = false) {
    if (ti < tend) {
      const int rt0 = r0 + Ri * HV_R, ct0 = r0 + Ci * HV_C;
      const zdf *src = A + rt0 + tr + lda * (ct0 + tc);
      zdf *dst = tiles + buf * (HV_C * HV_LD) + tc * HV_LD + tr;
      zdf *vdst = vecs + buf * (HV_R + HV_C) + tid;
      const int k = tid < HV_R ? rt0 + tid : ct0 + tid - HV_R;
      if (rt0 + HV_R <= n) {  // (every column of a full tile row exists)
#pragma unroll
        for (int j = 0; j < HV_C / 4; ++j) cp_async16(dst + 4 * j * HV_LD, src + 4 * j * lda);
        if (first) dep_wait();
        if (tid < HV_R + HV_C) cp_async16(vdst, A + k + lda * i);
      } else {
#pragma unroll
        for (int j = 0; j < HV_C / 4; ++j) {
          const bool ok = rt0 + tr < n && ct0 + tc + 4 * j < n;
          cp_async16(dst + 4 * j * HV_LD, ok ? (const void *)(src + 4 * j * lda) : (const void *)A, ok);
        }
        if (first) dep_wait();
        if (tid < HV_R + HV_C) cp_async16(vdst, k < n ? (const void *)(A + k + lda * i) : (const void *)A, k < n);
      }
      ++ti;
      if (++Ci > 2 * Ri + 1) {
        ++Ri;
        Ci = 0;
      }
    }
    cp_async_commit();
  };
  issue(0, true);
  zdf y = cz<df>();  // row sum (warps 0-3)
  zdf *Pm = Pb + b * sP;
  for (int buf = 0; t < tend; ++t, buf ^= 1) {
    cp_async_wait0();
    __syncthreads();  // this tile has landed, the other buffer is free
    issue(buf ^ 1);
    if (t + 1 == tend) dep_go();
    const zdf *tl = tiles + buf * (HV_C * HV_LD);
    const zdf *vl = vecs + buf * (HV_R + HV_C);
    const int off = HV_C * (Cc - 2 * R);  // >= 0 on the diagonal: entry (r, c) is below it for r > c + off
    if (warp < 4) {
      const int r = warp * 16 + (lane & 15), cb = lane & 16;
      const zdf *vc = vl + HV_R + cb, *ta = tl + cb * HV_LD + r;
      auto vec = [&](int k) { return vc[k]; };
      if (off < 0)
        df_block<false>(y, [&](int k) { return ta[k * HV_LD]; }, vec);
      else
        df_block<false>(y, [&](int k) { return r >= cb + k + off ? ta[k * HV_LD] : cz<df>(); }, vec);
      y = cfin(y);
      if (off == HV_C || t + 1 == tend) {  // the row sums end here
        y = cadd(y, zdf{shfl_xor_real(y.re, 16), shfl_xor_real(y.im, 16)});
        int first, nseg;
        hv_slots(R, run, first, nseg);
        const int row = r0 + R * HV_R + r;
        if (lane < 16 && row < n) Pm[(int64_t)(x - first) * ldp + row] = y;
        y = cz<df>();
      }
    } else {
      const int c = (warp - 4) * 8 + (lane & 7), rb = (lane >> 3) * 16;
      const zdf *vr = vl + rb, *ta = tl + c * HV_LD + rb;
      zdf s = cz<df>();
      auto vec = [&](int k) { return vr[k]; };
      if (off < 0)
        df_block<true>(s, [&](int k) { return ta[k]; }, vec);
      else
        df_block<true>(s, [&](int k) { return rb + k > c + off ? ta[k] : cz<df>(); }, vec);
      s = cfin(s);
      // over the four row groups: lanes below 16 end up with the real part, the others with the imaginary part
      const bool im = lane >= 16;
      df q = df_add(im ? s.im : s.re, shfl_xor_real(im ? s.re : s.im, 16));
      q = df_add(q, shfl_xor_real(q, 8));
      const df qi = shfl_xor_real(q, 16);
      const int col = r0 + Cc * HV_C + c;
      if (lane < 8 && col < n) Pm[(int64_t)(2 * nt + R) * ldp + col] = zdf{q, qi};
    }
    if (++Cc > 2 * R + 1) {
      ++R;
      Cc = 0;
    }
  }
  cp_async_wait0();
}

// ---- the work between two mat-vecs
// What the row work of panel column i reads.  Rows r >= col = i + 1; the
// mat-vec's partials of row r lie in `slots` slots of P: one per tile row /
// column of 32 (k_hemv_lower), or (double-float form) the runs of its tile row
// and the tile rows from its own on.
template <class R>
struct PanelCol {
  const C<R> *A, *W, *P;
  int64_t lda, ldp;
  int n, i, k0, jj, next, nt, run;  // next: column i + 1 belongs to the same panel
  __device__ __forceinline__ PanelCol(const C<R> *A_, const C<R> *W_, const C<R> *P_, int64_t lda_, int64_t ldp_, int n_,
                                      int i_, int k0_, int jj_, int next_, int sms)
      : A(A_), W(W_), P(P_), lda(lda_), ldp(ldp_), n(n_), i(i_), k0(k0_), jj(jj_), next(next_) {
    nt = cdiv_dev(n - i - 1, std::is_same<R, double>::value ? hl_tile(n - i - 1) : HV_R);
    run = std::is_same<R, double>::value ? 1 : hv_run(n - i - 1, jj, sms);
  }
  // the number of slots of row r: 0 .. nseg-1, then from nseg + skip on
  __device__ __forceinline__ int slots(int r, int &nseg, int &skip) const {
    if constexpr (std::is_same<R, double>::value) {
      nseg = nt;
      skip = 0;
      return nt;
    } else {
      int first;
      const int Rt = (r - i - 1) / HV_R;
      hv_slots(Rt, run, first, nseg);
      skip = 2 * nt + Rt - nseg;
      return nseg + nt - Rt;
    }
  }
};
// What one lane (sub = 0 .. 7 of the row's eight) reads of row r: its slots
// and panel columns sub, sub + 8, ..., and, in lane 0, v and column i + 1.
constexpr int CT_TPR = 8;
template <class R>
struct PanelRow {
  C<R> p[4], w[4], v[4], vi, a;
  // the mat-vec's results
  __device__ __forceinline__ void load_p(const PanelCol<R> &c, int r, int sub) {
    const bool in = r < c.n;
    int nseg, skip;
    const int nch = c.slots(in ? r : c.i + 1, nseg, skip);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = sub + CT_TPR * u;
      p[u] = in && k < nch ? c.P[r + (int64_t)(k + (k >= nseg ? skip : 0)) * c.ldp] : cz<R>();
    }
  }
  // what was there before it (loaded before dep_wait, too)
  __device__ __forceinline__ void load_old(const PanelCol<R> &c, int r, int sub) {
    const bool in = r < c.n;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = sub + CT_TPR * u;
      w[u] = in && k < c.jj ? load_l2(&c.W[r + c.lda * k]) : cz<R>();
      v[u] = in && k < c.jj ? load_l2(&c.A[r + c.lda * (c.k0 + k)]) : cz<R>();
    }
    const bool own = in && sub == 0;
    vi = own ? load_l2(&c.A[r + c.lda * c.i]) : cz<R>();
    a = own && c.next ? load_l2(&c.A[r + c.lda * (c.i + 1)]) : cz<R>();
  }
  // y = (mat-vec) - W x1 - V x2 and nxt = the panel columns' part of column
  // i + 1's update (x1, x2, row i + 1 of V and W conjugated in shared memory),
  // summed over the row's eight lanes
  __device__ __forceinline__ void sums(const PanelCol<R> &c, int r, int sub, const C<R> *x1, const C<R> *x2,
                                       const C<R> *nv, const C<R> *nw, C<R> &y, C<R> &nxt) const {
    y = cadd(cadd(p[0], p[1]), cadd(p[2], p[3]));
    nxt = cz<R>();
    int nseg, skip;
    const int nch = c.slots(r < c.n ? r : c.i + 1, nseg, skip);
    for (int ch = sub + 4 * CT_TPR; ch < nch; ch += 4 * CT_TPR) {
      C<R> t[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = ch + CT_TPR * u;
        t[u] = r < c.n && k < nch ? c.P[r + (int64_t)(k + (k >= nseg ? skip : 0)) * c.ldp] : cz<R>();
      }
      y = cadd(y, cadd(cadd(t[0], t[1]), cadd(t[2], t[3])));
    }
    C<R> acc = cz<R>();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = sub + CT_TPR * u;
      if (CT_TPR * u >= c.jj) break;
      if (k < c.jj) {
        cmac(acc, w[u], x1[k]);
        cmac(acc, v[u], x2[k]);
        if (c.next) {
          cmac(nxt, v[u], nw[k]);
          cmac(nxt, w[u], nv[k]);
        }
      }
    }
    y = csub(y, cfin(acc));
    nxt = cfin(nxt);
    group8_sum(y, nxt);
  }
};
// row i + 1 of V and W (conjugated) and, the mat-vec's, x1 = V^H v, x2 = W^H v
// into shared memory
template <class R>
__device__ __forceinline__ void panel_next(const PanelCol<R> &c, C<R> *nv, C<R> *nw) {
  if (c.next)
    for (int k = threadIdx.x; k < c.jj; k += blockDim.x) {
      nv[k] = cconj(load_l2(&c.A[c.i + 1 + c.lda * (c.k0 + k)]));
      nw[k] = cconj(load_l2(&c.W[c.i + 1 + c.lda * k]));
    }
}
template <class R>
__device__ __forceinline__ void panel_x(const PanelCol<R> &c, const C<R> *X, C<R> *x1, C<R> *x2) {
  for (int k = threadIdx.x; k < c.jj; k += blockDim.x) {
    x1[k] = X[k];
    x2[k] = X[c.jj + k];
  }
}
constexpr int ROWSUM_BYTES = 32;  // the larger of the two forms
static_assert(sizeof(RowSum<df>) == ROWSUM_BYTES && sizeof(RowSum<double>) <= ROWSUM_BYTES, "partial-sum slots");

// Large trailing blocks: the row work of column i on the whole chip.
//   w0 = tau (y - W x1 - V x2) into column jj of W, column i + 1 less the panel
//   columns' part, and one partial of w0^H v per block.
// k_colstep then only completes w and forms the next reflector.
template <class R>
constexpr int wp_threads = std::is_same<R, double>::value ? 128 : 256;  // FP64: spread over more SMs' FP64 pipes
template <class R>
__global__ void __launch_bounds__(wp_threads<R>) k_wpart(C<R> *Ab, int64_t lda, int64_t sA, C<R> *Wb, int64_t sW,
                                                         const C<R> *Pb, int64_t sP, int64_t ldp, const int *nvec, int i,
                                                         int k0, int jj, int next, int sms, const C<R> *X, int ldx,
                                                         const C<R> *taub, RowSum<R> *partb, int64_t spart) {
  constexpr int NW = wp_threads<R> / 32;
  __shared__ C<R> x1[32], x2[32], nv[32], nw[32];
  __shared__ RowSum<R> red[NW];
  const int b = blockIdx.y;
  const int n = nvec[b];
  const int col = i + 1;
  const int rb = col + blockIdx.x * NW * 4;
  if (rb >= n) {
    dep_wait();
    return;
  }
  C<R> *A = Ab + b * sA;
  C<R> *W = Wb + b * sW;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = tid % CT_TPR;
  const PanelCol<R> pc(A, W, Pb + b * sP, lda, ldp, n, i, k0, jj, next, sms);
  const int r = rb + tid / CT_TPR;
  PanelRow<R> q;
  q.load_old(pc, r, sub);
  const C<R> tau = load_l2(&taub[b]);
  panel_next(pc, nv, nw);
  dep_wait();
  q.load_p(pc, r, sub);
  panel_x(pc, X + b * ldx, x1, x2);
  dep_go();
  __syncthreads();
  C<R> y, nxt;
  RowSum<R> dot;
  dot.zero();
  q.sums(pc, r, sub, x1, x2, nv, nw, y, nxt);
  RowSum<R> *part = partb + b * spart;
  if (sub == 0 && r < n) {
    const C<R> w = cmul(tau, y);
    W[r + lda * jj] = w;
    if (next) A[r + lda * col] = csub(q.a, nxt);
    dot.add_product(w, q.vi);
    if (r == col) *(C<R> *)&part[0] = w;  // w0(i+1)
  }
  dot.rows4();
  if (lane == 0) red[warp] = dot;
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int k = 1; k < NW; ++k) dot.add(red[k]);
    part[1 + blockIdx.x] = dot;
  }
}

// One panel column's scalar and row work, one cluster of CTAs per matrix (rows
// are dealt to the CTAs' warps in groups of 4).  With do_w != 0, for column i
// (its mat-vec partials in P, the products x1 = V^H v and x2 = W^H v in X):
//   w0 = tau (y - W x1 - V x2),  alpha = -1/2 tau (w0^H v),  w = w0 + alpha v
//   (column jj of W); do_w = 2: w0, the panel columns' part of column i + 1
//   and the nparts partials of w0^H v were formed by k_wpart;
// with do_next, for column i + 1 = col of the same panel (do_w = 0: the
// panel's first column):
//   A(col:n, col) -= V W(col,:)^H + W V(col,:)^H over the panel columns 0..jj,
//   d, the reflector (zlarfg: beta, tau, v = [1; x / (alpha - beta)]) and v
//   written back in place.
// The two global sums (w0^H v and |x|^2) cross the CTAs through distributed
// shared memory: each warp writes its part into every CTA of the cluster and
// passes the cluster barrier (0.2-0.3 us).  Bound by latency: the loads of a
// row (partial slots, panel columns, v, the next column) are all issued at
// once, ahead of the first barrier; a row's w, v and next-column entry stay in
// shared memory between the phases (rows past CT_CAP of a CTA: in global
// memory).  Eight threads share a row, each summing every eighth partial slot
// and panel column.  Measured, one matrix, 16 panel columns, a column's launches
// besides the mat-vec: four before (column update, reflector, panel products,
// corrections; 7-12 us each, mostly FP64 reductions, divisions and square
// roots), now 9.3 us at n = 84 (one launch), 11.5 us at n = 1092 and 13.3 us at
// n = 4764 (with k_wpart).  w0^H v in three floats and alpha in FP64, instead of
// products rounded to double-float, take 0.9% of a pass (n = 2604 x 4).
constexpr int CT_CLUSTER = 16;           // largest cluster (non-portable size, where it can be placed)
constexpr int CT_CAP = 512;              // rows of a CTA kept in shared memory
constexpr int CT_NW = TR_NT / 32;        // warps
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of a shared variable of this CTA in CTA `rank` of the cluster
template <class T>
__device__ __forceinline__ T *cluster_ptr(T *p, int rank) {
  uint64_t out;
  asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"((uint64_t)p), "r"(rank));
  return (T *)out;
}

template <class R>
__global__ void __launch_bounds__(TR_NT) k_colstep(C<R> *Ab, int64_t lda, int64_t sA, C<R> *Wb, int64_t sW,
                                                   const C<R> *Pb, int64_t sP, int64_t ldp, const int *nvec, int i,
                                                   int k0, int jj, int do_w, int do_next, int sms, const C<R> *X,
                                                   int ldx, const RowSum<R> *partb, int64_t spart, C<R> *taub, double *dd,
                                                   double *ee, z64 *tau64, int64_t sd) {
  typedef Sum<R> S;
  typedef typename S::T T;
  __shared__ C<R> cw[CT_CAP], cv[CT_CAP], ca[CT_CAP];
  __shared__ C<R> x1[32], x2[32], nv[32], nw[32];
  // written by the warps of the whole cluster
  __shared__ RowSum<R> in_wv[CT_CLUSTER * CT_NW];
  __shared__ T in_sq[CT_CLUSTER * CT_NW];
  __shared__ int in_e[CT_CLUSTER * CT_NW];
  __shared__ C<R> in_w, in_alpha;
  // results of the CTA's first warp
  __shared__ C<R> s_alpha, s_wn, s_scale;
  __shared__ int s_skip, s_e;
  const int rank = blockIdx.x, CS = gridDim.x;  // the cluster spans gridDim.x
  const int b = blockIdx.y;
  const int n = nvec[b];
  const int col = i + 1;
  if (do_w != 1 || col >= n) dep_wait();
  if (col >= n) return;
  cluster_arrive();  // distributed shared memory may be written once every CTA has started
  bool started = false;
  C<R> *A = Ab + b * sA;
  C<R> *W = Wb + b * sW;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // row of local index l (groups of 4 rows dealt to the CTAs in turn)
  auto row_of = [&](int l) { return col + ((l >> 2) * CS + rank) * 4 + (l & 3); };
  const bool cached = do_w == 1;  // w0, v and column col are in shared memory
  C<R> alpha = cz<R>(), wn = cz<R>();
  // alpha (over the first warp) and w(i+1): v(i+1) = 1
  auto finish_alpha = [&](const RowSum<R> &part, C<R> w0, double2 t) {
    const C<R> al = minus_half_product(part, z64{t.x, t.y});
    if (lane == 0) {
      s_alpha = al;
      s_wn = cadd(w0, al);
    }
  };
  // tau of column i in FP64 (written by the launch that formed its reflector)
  const double2 *tau_i = (const double2 *)&tau64[b * sd + (i < 0 ? 0 : i)];
  if (do_w == 1) {
    const PanelCol<R> pc(A, W, Pb + b * sP, lda, ldp, n, i, k0, jj, do_next, sms);
    const int sub = lane % CT_TPR;
    PanelRow<R> q;
    int l = warp * 4 + lane / CT_TPR;
    q.load_old(pc, row_of(l), sub);
    const C<R> tau = load_l2(&taub[b]);
    const double2 t64 = __ldcg(tau_i);
    panel_next(pc, nv, nw);
    dep_wait();
    q.load_p(pc, row_of(l), sub);
    panel_x(pc, X + b * ldx, x1, x2);
    __syncthreads();
    RowSum<R> dot;
    dot.zero();
    C<R> wfirst = cz<R>();
    while (row_of(l & ~3) < n) {  // (uniform over the warp)
      const int r = row_of(l);
      C<R> y, nxt;
      q.sums(pc, r, sub, x1, x2, nv, nw, y, nxt);
      if (sub == 0 && r < n) {
        const C<R> w = cmul(tau, y);
        const C<R> a = csub(q.a, nxt);
        if (l < CT_CAP) {
          cw[l] = w;
          cv[l] = q.vi;
          ca[l] = a;
        } else {
          W[r + lda * jj] = w;
          if (do_next) A[r + lda * col] = a;
        }
        dot.add_product(w, q.vi);
        if (l == 0) wfirst = w;
      }
      l += 4 * CT_NW;
      if (row_of(l & ~3) < n) {
        q.load_old(pc, row_of(l), sub);
        q.load_p(pc, row_of(l), sub);
      }
    }
    // w0^H v: lanes 0, 8, 16, 24 of each warp, then all warps of the cluster
    dot.rows4();
    RowSum<R> part;
    part.re = shfl_real(dot.re, 0);
    part.im = shfl_real(dot.im, 0);
    const C<R> wf{shfl_real(wfirst.re, 0), shfl_real(wfirst.im, 0)};
    cluster_wait();
    started = true;
    if (lane < CS) {
      *cluster_ptr(&in_wv[rank * CT_NW + warp], lane) = part;
      if (rank == 0 && warp == 0) *cluster_ptr(&in_w, lane) = wf;
    }
    cluster_arrive();
    cluster_wait();
    if (warp == 0) {
      RowSum<R> mine;
      mine.zero();
      for (int k = lane; k < CS * CT_NW; k += 32) mine.add(in_wv[k]);
      finish_alpha(mine, in_w, t64);
    }
    __syncthreads();
  } else if (do_w == 2) {
    if (warp == 0) {
      const RowSum<R> *part = partb + b * spart;
      const double2 t64 = __ldcg(tau_i);
      const int nparts = cdiv_dev(n - col, wp_threads<R> / CT_TPR);
      RowSum<R> mine;
      mine.zero();
      for (int k = lane; k < nparts; k += 32) mine.add(part[1 + k]);
      finish_alpha(mine, *(const C<R> *)&part[0], t64);
    }
    __syncthreads();
  }
  if (do_w) {
    alpha = s_alpha;
    wn = cconj(s_wn);
  }
  // ---- one thread per row: w completed, column `col` updated
  float big = 0.f;
  for (int l = tid; row_of(l) < n; l += TR_NT) {
    const int r = row_of(l);
    const bool held = l < CT_CAP;
    C<R> a = cz<R>();
    if (do_next) a = held && cached ? ca[l] : A[r + lda * col];
    if (do_w) {
      const C<R> v = held && cached ? cv[l] : A[r + lda * i];
      C<R> w = held && cached ? cw[l] : W[r + lda * jj];
      cmac(w, alpha, v);
      w = cfin(w);
      W[r + lda * jj] = w;
      if (do_next) {
        C<R> acc = w;  // conj(v(i+1)) = 1
        cmac(acc, v, wn);
        a = csub(a, cfin(acc));
      }
    }
    if (do_next) {
      if (r == col) a.im = RT<R>::zero();
      if (r == col + 1) s_scale = a;  // alpha of the reflector (rank 0; read below, before it is reused)
      if (r >= col + 2) big = fmaxf(big, magnitude(a));
      if (held)
        ca[l] = a;
      else
        A[r + lda * col] = a;
    }
  }
  if (!do_next || col == n - 1) {  // the panel's last column, or no reflector: the matrix ends here
    if (do_next && rank == 0 && tid == 0) {
      A[col + lda * col] = ca[0];
      dd[b * sd + col] = RT<R>::to(ca[0].re);
      tau64[b * sd + col] = z64{0.0, 0.0};
      ee[b * sd + col] = 0.0;
      taub[b] = cz<R>();
    }
    if (!started) cluster_wait();
    return;
  }
  // |x|^2.  Double-float: of the values scaled by the warp's largest exponent
  // (the float square of a small entry would underflow)
  __syncwarp();
  int e = 0;
  if constexpr (!std::is_same<R, double>::value)
    e = min(max((int)(__reduce_max_sync(0xffffffffu, __float_as_uint(big)) >> 23) - 127, -120), 120);
  T sq = S::zero();
  for (int l = tid; row_of(l) < n; l += TR_NT) {
    const int r = row_of(l);
    if (r < col + 2) continue;
    const C<R> a = prescale(l < CT_CAP ? ca[l] : A[r + lda * col], e);
    sq = S::add(sq, S::add(S::mul(a.re, a.re), S::mul(a.im, a.im)));
  }
  __syncwarp();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq = S::add(sq, S::shfl_xor(sq, o));
  if (!started) cluster_wait();
  if (lane < CS) {
    *cluster_ptr(&in_sq[rank * CT_NW + warp], lane) = sq;
    *cluster_ptr(&in_e[rank * CT_NW + warp], lane) = e;
    // (row col + 1 is the second thread's of rank 0)
    if (rank == 0 && warp == 0) *cluster_ptr(&in_alpha, lane) = s_scale;
  }
  cluster_arrive();
  cluster_wait();
  Reflector<R> f;
  if (warp == 0) {
    int emax = 0;
    if constexpr (!std::is_same<R, double>::value) {
      int el = -120;
      for (int k = lane; k < CS * CT_NW; k += 32) el = max(el, in_e[k]);
      emax = __reduce_max_sync(0xffffffffu, el);
    }
    T v = S::zero();
    for (int k = lane; k < CS * CT_NW; k += 32) {
      if constexpr (!std::is_same<R, double>::value) {
        const int d2 = 2 * (in_e[k] - emax);
        v = S::add(v, tf_scale(in_sq[k], d2 < -126 ? 0.f : pow2_clamped(d2)));
      } else {
        v = S::add(v, in_sq[k]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = S::add(v, S::shfl_xor(v, o));
    f = reflector_scalars(v, emax, in_alpha);
    if (lane == 0) {
      s_scale = f.scale;
      s_skip = f.skip;
      s_e = f.e;
    }
  }
  __syncthreads();
  dep_go();
  const C<R> sc = s_scale;
  const int skip = s_skip, pe = s_e;
  for (int l = tid; row_of(l) < n; l += TR_NT) {
    const int r = row_of(l);
    C<R> a = l < CT_CAP ? ca[l] : A[r + lda * col];
    if (r == col + 1) a = C<R>{RT<R>::from(1.0), RT<R>::zero()};
    if (r >= col + 2 && !skip) a = cmul(prescale(a, pe), sc);
    A[r + lda * col] = a;
  }
  if (rank == 0 && warp == 0) {
    // four conversions to FP64, one per lane
    const T q = lane == 0 ? S::from(ca[0].re) : lane == 1 ? f.beta : lane == 2 ? f.t_re : f.t_im;
    const double x = S::to(q) * __hiloint2double((1023 + (lane == 1 ? f.e : 0)) << 20, 0);
    if (lane == 0) {
      dd[b * sd + col] = x;
      taub[b] = f.tau;
    }
    if (lane == 1) ee[b * sd + col] = x;
    if (lane == 2) tau64[b * sd + col].re = x;
    if (lane == 3) tau64[b * sd + col].im = x;
  }
}

// Trailing update A(k1:n, k1:n) -= V W^H + W V^H (full square), K = jb.
// Tiles of 32 x 32 (2 x 2 per thread): with 64 x 64 a trailing block of a few
// hundred rows had fewer tiles than SMs, and one of order 52 a single one
// (FP64 pipe: 2 multiply-adds per SM and clock; n = 84 265 -> 72 us a launch,
// n = 1092 343 -> 167 us, two of n = 2604 1169 -> 1017 us).
constexpr int HK_T = 32, HK_K = 16, HK_P = HK_T / 16;
template <class R>
__global__ void __launch_bounds__(256) k_her2k(C<R> *Ab, int64_t lda, int64_t sA, const C<R> *Wb, int64_t sW,
                                               const int *nvec, int k0, int jb) {
  __shared__ C<R> sVr[HK_K][HK_T], sWr[HK_K][HK_T], sVc[HK_K][HK_T], sWc[HK_K][HK_T];
  const int b = blockIdx.z;
  const int n = nvec[b];
  const int k1 = k0 + jb;
  if (blockIdx.x < blockIdx.y) return;  // only the lower triangle is kept
  const int r0 = k1 + blockIdx.x * HK_T, c0 = k1 + blockIdx.y * HK_T;
  if (r0 >= n || c0 >= n) return;
  C<R> *A = Ab + b * sA;
  const C<R> *W = Wb + b * sW;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  C<R> acc[HK_P][HK_P];
#pragma unroll
  for (int p = 0; p < HK_P; ++p)
#pragma unroll
    for (int q = 0; q < HK_P; ++q) acc[p][q] = cz<R>();
  const int jmax = min(jb, n - 1 - k0);  // reflectors that exist in this matrix
  for (int kc = 0; kc < jmax; kc += HK_K) {
    for (int e = threadIdx.x; e < HK_K * HK_T; e += 256) {
      int x = e % HK_T, y = e / HK_T;
      int k = kc + y;
      int rr = r0 + x, cc = c0 + x;
      bool ok = k < jmax;
      sVr[y][x] = (ok && rr < n) ? A[rr + lda * (k0 + k)] : cz<R>();
      sWr[y][x] = (ok && rr < n) ? W[rr + lda * k] : cz<R>();
      sVc[y][x] = (ok && cc < n) ? cconj(A[cc + lda * (k0 + k)]) : cz<R>();
      sWc[y][x] = (ok && cc < n) ? cconj(W[cc + lda * k]) : cz<R>();
    }
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < HK_K; ++k) {
      C<R> vr[HK_P], wr[HK_P], vc[HK_P], wc[HK_P];
#pragma unroll
      for (int p = 0; p < HK_P; ++p) {
        vr[p] = sVr[k][tx + 16 * p];
        wr[p] = sWr[k][tx + 16 * p];
        vc[p] = sVc[k][ty + 16 * p];
        wc[p] = sWc[k][ty + 16 * p];
      }
#pragma unroll
      for (int p = 0; p < HK_P; ++p)
#pragma unroll
        for (int q = 0; q < HK_P; ++q) {
          cmac(acc[p][q], vr[p], wc[q]);
          cmac(acc[p][q], wr[p], vc[q]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < HK_P; ++p)
#pragma unroll
    for (int q = 0; q < HK_P; ++q) {
      int rr = r0 + tx + 16 * p, cc = c0 + ty + 16 * q;
      if (rr < n && cc < n) {
        C<R> *x = &A[rr + lda * cc];
        *x = csub(*x, cfin(acc[p][q]));
      }
    }
}

// Persistent hemv blocks: bps per SM of the current device (at most HL_BPS,
// the residency the kernel is compiled for).
static int hemv_blocks(int bps) { return device_sms() * std::max(1, std::min(bps, HL_BPS)); }

// Clusters of 16 CTAs are beyond the portable size, the mat-vec's tiles beyond
// 48 KB of shared memory: opted in once per device.  *cluster: the column step's
// largest cluster there, 16 or what the device (a partition of it) can place, at
// least the portable 8; PARPHOM_GPU_CLUSTER caps it.
template <class R>
static cudaError_t prepare_colstep(int *cluster) {
  static std::mutex mu;
  static int largest[PP_MAX_DEVICES] = {};
  const int dev = device_index();
  {
    std::lock_guard<std::mutex> g(mu);
    int c = dev >= 0 ? largest[dev] : 0;
    if (c == 0) {
      c = 8;
      if (cudaFuncSetAttribute(k_colstep<R>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(CT_CLUSTER);
        cfg.blockDim = dim3(TR_NT);
        int most = 0;
        if (cudaOccupancyMaxPotentialClusterSize(&most, k_colstep<R>, &cfg) == cudaSuccess)
          while (c < CT_CLUSTER && 2 * c <= most) c *= 2;
      }
      cudaGetLastError();
      if (std::is_same<R, df>::value)
        PP_CUDA_TRY(cudaFuncSetAttribute(k_hemv_df, cudaFuncAttributeMaxDynamicSharedMemorySize, HV_SMEM));
      if (dev >= 0) largest[dev] = c;
    }
    *cluster = c;
  }
  if (const char *v = getenv("PARPHOM_GPU_CLUSTER")) {
    const int cap = atoi(v);
    while (cap > 0 && *cluster > cap) *cluster /= 2;
  }
  return cudaSuccess;
}

// One column step; the cluster has a CTA per 8 rows, at most CT_CLUSTER, and
// fewer where the whole batch would not run at once (two CTAs fit an SM; 64
// matrices of order 444, FP64: 48 us a column with clusters of 16, 29 us with
// clusters of 4).  Past CT_SPLIT rows the row work
// goes to the whole chip first (k_wpart): one cluster works through CT_SPLIT
// rows in one pass, and more passes cost more than the extra launch (both
// launches against one: 11.5 us / 13.3 us at n = 1092, 13.2 us / 34.9 us at
// n = 4764; FP64 form 12.4 us / 22.4 us at n = 1092).
constexpr int CT_SPLIT = CT_CLUSTER * CT_NW * 4;
template <class R>
static cudaError_t launch_colstep(EigWork &w, int i, int k0, int jj, int do_w, int do_next, int cluster, cudaStream_t s) {
  const int rows = w.nmax - i - 1;
  const int64_t sW = (int64_t)w.lda * w.nb, sP = (int64_t)w.nchunk * w.lda;
  if (do_w && rows > CT_SPLIT) {
    do_w = 2;
    cudaError_t e = cudaSuccess;
    PP_KT(KT_COLSTEP, s, (e = launch_dep(k_wpart<R>, dim3(cdiv(rows, wp_threads<R> / CT_TPR), w.B), wp_threads<R>, 0, 0, true,
                                         s, (C<R> *)w.A, w.lda, w.sA, (C<R> *)w.W, sW, (const C<R> *)w.P, sP, w.lda, w.nvec,
                                         i, k0, jj, do_next, device_sms(), (const C<R> *)w.X, 2 * w.nb,
                                         (const C<R> *)w.scal, (RowSum<R> *)w.part,
                                         w.spart * ROWSUM_BYTES / (int)sizeof(RowSum<R>))));
    PP_CUDA_TRY(e);
    count_launch(1);
  }
  int cs = 1;
  while (cs < cluster && cs * 8 < rows && cs * std::max(w.batch, w.B) <= device_sms()) cs *= 2;
  cudaError_t e = cudaSuccess;
  PP_KT(KT_COLSTEP, s, (e = launch_dep(k_colstep<R>, dim3(cs, w.B), TR_NT, 0, cs, do_w != 0, s, (C<R> *)w.A, w.lda, w.sA,
                                       (C<R> *)w.W, sW, (const C<R> *)w.P, sP, w.lda, (const int *)w.nvec, i, k0, jj, do_w,
                                       do_next, device_sms(), (const C<R> *)w.X, 2 * w.nb, (const RowSum<R> *)w.part,
                                       w.spart * ROWSUM_BYTES / (int)sizeof(RowSum<R>), (C<R> *)w.scal, w.d, w.e, w.tau,
                                       (int64_t)w.nmax)));
  count_launch(1);
  return e;
}

// Whether a matrix of the batch has a trailing block of 1 .. HL_SMALL rows past
// column i (one that has ended has none: the larger ones carry no empty launch).
static bool any_small(const EigWork &w, int i) {
  auto small = [&](int n) { return n - i - 1 > 0 && n - i - 1 <= HL_SMALL; };
  return w.orders ? std::any_of(w.orders, w.orders + w.B, small) : small(w.nmax);
}

template <class R>
cudaError_t tridiagonalize(EigWork &w, cudaStream_t s) {
  C<R> *A = (C<R> *)w.A;
  C<R> *W = (C<R> *)w.W;
  C<R> *P = (C<R> *)w.P;
  const int B = w.B, nmax = w.nmax, nb = w.nb;
  const int64_t lda = w.lda, sA = w.sA, sW = (int64_t)w.lda * nb, sP = (int64_t)w.nchunk * w.lda;
  int cluster = 1;
  PP_CUDA_TRY(prepare_colstep<R>(&cluster));
  if (w.tcErr) PP_CUDA_TRY(cudaMemsetAsync(w.tcErr, 0, sizeof(int) * B, s));
  for (int k0 = 0; k0 < nmax; k0 += nb) {
    const int jb = min(nb, nmax - k0);
    PP_CUDA_TRY(launch_colstep<R>(w, k0 - 1, k0, 0, 0, 1, cluster, s));  // the panel's first column
    for (int jj = 0; jj < jb; ++jj) {
      const int i = k0 + jj;
      if (i >= nmax - 1) break;
      if constexpr (std::is_same<R, df>::value) {
        // (a smaller matrix of the batch may have more, shorter runs)
        const int nt = cdiv(nmax - i - 1, HV_R);
        const int gx = hv_dots(jj) + std::min(nt * (nt + 1), hv_ctas(jj, device_sms()));
        cudaError_t e = cudaSuccess;
        PP_KT(KT_HEMV, s, (e = launch_dep(k_hemv_df, dim3(gx, B), HV_NT, HV_SMEM, 0, true, s, A, lda, sA, w.nvec, i, P, sP,
                                          lda, W, sW, k0, jj, (C<R> *)w.X, 2 * nb, device_sms())));
        PP_CUDA_TRY(e);
        count_launch(1);
      } else {
        // (the tile follows each matrix's own order: a batch that has both kinds runs both kernels)
        const int rows = nmax - i - 1;
        if (rows > HL_SMALL) {
          const int nt = cdiv(rows, HL_T);
          const int gx = hl_dots(jj, HL_T) + std::min(nt * (nt + 1) / 2, hemv_blocks(w.hemv_bps));
          cudaError_t e = cudaSuccess;
          PP_KT(KT_HEMV, s, (e = launch_dep(k_hemv_lower<HL_T>, dim3(gx, 1, B), 4 * HL_T, 0, 0, true, s, A, lda, sA, w.nvec,
                                            i, P, sP, lda, W, sW, k0, jj, (C<R> *)w.X, 2 * nb)));
          PP_CUDA_TRY(e);
          count_launch(1);
        }
        if (any_small(w, i)) {
          const int nt = cdiv(std::min(rows, HL_SMALL), HL_TS);
          const int gx = hl_dots(jj, HL_TS) + nt * (nt + 1) / 2;
          cudaError_t e = cudaSuccess;
          PP_KT(KT_HEMV, s, (e = launch_dep(k_hemv_lower<HL_TS>, dim3(gx, 1, B), 4 * HL_TS, 0, 0, true, s, A, lda, sA,
                                            w.nvec, i, P, sP, lda, W, sW, k0, jj, (C<R> *)w.X, 2 * nb)));
          PP_CUDA_TRY(e);
          count_launch(1);
        }
      }
      PP_CUDA_TRY(launch_colstep<R>(w, i, k0, jj, 1, jj + 1 < jb ? 1 : 0, cluster, s));
    }
    const int k1 = k0 + jb;
    if (k1 < nmax) {
      if (std::is_same<R, df>::value && w.tcS && tc_enabled()) {
        PP_CUDA_TRY(her2k_tc(w, k0, jb, s));
      } else {
        const int m = nmax - k1;
        dim3 g(cdiv(m, HK_T), cdiv(m, HK_T), B);
        PP_KT(KT_HER2K, s, (k_her2k<R><<<g, 256, 0, s>>>(A, lda, sA, W, sW, w.nvec, k0, jb)));
        count_launch(1);
      }
    }
  }
  return cudaGetLastError();
}

// ===========================================================================
// Stage 2: eigenvalues of the tridiagonal matrix (FP64 bisection)
// ===========================================================================
// Gerschgorin interval, pivmin and the index range of the wanted eigenvalues
// (one block per matrix; the extrema do not depend on the order of the rows).
constexpr int TD_NT = 256;
__global__ void __launch_bounds__(TD_NT) k_tdprep(const double *dd, const double *ee, int64_t sd, const int *nvec,
                                                  char range, double vl, double vu, int64_t il, int64_t iu, int64_t *rng,
                                                  double *tinfo, int64_t *info, const int *tcerr) {
  __shared__ double sgl[TD_NT / 32], sgu[TD_NT / 32], se2[TD_NT / 32];
  __shared__ int scount[2];
  const int b = blockIdx.x;
  const int n = nvec[b];
  const double *d = dd + b * sd;
  const double *e = ee + b * sd;
  double gl = d[0], gu = d[0], emax2 = 0.0;
  for (int k = threadIdx.x; k < n; k += TD_NT) {
    const double off = (k > 0 ? fabs(e[k - 1]) : 0.0) + (k < n - 1 ? fabs(e[k]) : 0.0);
    gl = fmin(gl, d[k] - off);
    gu = fmax(gu, d[k] + off);
    if (k < n - 1) emax2 = fmax(emax2, e[k] * e[k]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, o));
    gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, o));
    emax2 = fmax(emax2, __shfl_xor_sync(0xffffffffu, emax2, o));
  }
  if ((threadIdx.x & 31) == 0) {
    sgl[threadIdx.x >> 5] = gl;
    sgu[threadIdx.x >> 5] = gu;
    se2[threadIdx.x >> 5] = emax2;
  }
  __syncthreads();
  for (int k = 0; k < TD_NT / 32; ++k) {
    gl = fmin(gl, sgl[k]);
    gu = fmax(gu, sgu[k]);
    emax2 = fmax(emax2, se2[k]);
  }
  const double ulp = DBL_EPSILON;
  const double safmin = DBL_MIN;
  double tnorm = fmax(fabs(gl), fabs(gu));
  double pivmin = safmin * fmax(1.0, emax2);
  const double fudge = 2.1;
  gl = gl - fudge * tnorm * ulp * n - fudge * 2.0 * pivmin;
  gu = gu + fudge * tnorm * ulp * n + fudge * 2.0 * pivmin;
  int64_t lo = 1, hi = n;
  if (range == 'I') {
    lo = il;
    hi = iu;
  } else if (range == 'V') {
    // eigenvalues in the half-open interval (vl, vu]: a count each in the first threads of two warps
    // local e^2 recomputed on the fly
    if (threadIdx.x == 0 || threadIdx.x == 32) {
      const double x = threadIdx.x == 0 ? vl : vu;
      double q = d[0] - x;
      if (fabs(q) <= pivmin) q = -pivmin;
      int c = q < 0.0;
      for (int k = 1; k < n; ++k) {
        q = d[k] - (e[k - 1] * e[k - 1]) / q - x;
        if (fabs(q) <= pivmin) q = -pivmin;
        c += q < 0.0;
      }
      scount[threadIdx.x / 32] = c;
    }
    __syncthreads();
    lo = scount[0] + 1;
    hi = scount[1];
  }
  if (threadIdx.x != 0) return;
  int64_t m = hi - lo + 1;
  if (m < 0) m = 0;
  rng[b * 8 + 0] = lo;
  rng[b * 8 + 1] = hi;
  rng[b * 8 + 2] = m;
  tinfo[b * 8 + 0] = gl;
  tinfo[b * 8 + 1] = gu;
  tinfo[b * 8 + 2] = tnorm;
  tinfo[b * 8 + 3] = pivmin;
  info[b] = (tcerr && tcerr[b]) ? PP_INFO_TIMEOUT : 0;
}

// FP64 Sturm count (the number of eigenvalues below x) of the tridiagonal
// scaled by a power of two to norm 1/2 .. 1, by the recurrence of the leading
// principal minors
//   p_{k+1} = (d_k - x) p_k - e_{k-1}^2 p_{k-1},
// a sign change per eigenvalue below x.  Like the quotient form q = p_{k+1} /
// p_k it is exact for entries perturbed by a few units in the last place, but
// a row costs one dependent multiply-add instead of a division (85 instead of
// 600 cycles of latency, 3 instead of ~20 operations on a pipe that takes 16
// cycles per warp operation).  Rows are taken MC_NB at a time, the pair (p_k,
// p_{k+1}) rescaled by a power of two after each block.  If a minor of the
// block falls below 2^-MC_LIM, the block is repeated row by row with a
// rescaling after each, and a vanishing minor replaced by -2^-MC_PIV p_k (a
// quotient of -2^-MC_PIV, as the quotient form does).  (The float and
// double-float counts keep the quotient form: their reciprocals take 40
// cycles, and the minors' checks cost more than that saves.)
constexpr int MC_NB = 8, MC_LIM = 700, MC_PIV = 400;
struct MinorCount {
  const double2 *t;     // d, e^2 in shared memory, or null:
  const double *d, *e;  // from global memory, to be scaled by sc
  double sc;
  __device__ __forceinline__ double step(int k, double x, double p0, double p1) const {
    double dk, e2;
    if (t) {
      dk = t[k].x;
      e2 = t[k - 1].y;
    } else {
      const double ek = e[k - 1] * sc;
      dk = d[k] * sc;
      e2 = ek * ek;
    }
    return fma(dk - x, p1, -(e2 * p0));
  }
  __device__ static __forceinline__ int expo(double p) { return ((__double2hiint(p) >> 20) & 2047) - 1023; }
  __device__ static __forceinline__ double scale(double p, int e) { return p * __hiloint2double((1023 + e) << 20, 0); }
  // the larger of the pair brought to exponent 0
  __device__ static __forceinline__ void rescale(double &p0, double &p1) {
    const int e = max(expo(p0), expo(p1));
    p0 = scale(p0, -e);
    p1 = scale(p1, -e);
  }
  __device__ static __forceinline__ void guard(double &p0, double &p1) {
    if (expo(p1) < expo(p0) - MC_PIV) p1 = -scale(p0, -MC_PIV);  // (zero: exponent -1023)
    rescale(p0, p1);
  }
  __device__ __forceinline__ int operator()(int n, double x) const {
    double p0 = 1.0, p1 = (t ? t[0].x : d[0] * sc) - x;
    guard(p0, p1);
    unsigned cnt = (unsigned)__double2hiint(p1) >> 31;
    auto rows = [&](int k, int k1) {
      for (; k < k1; ++k) {
        const double q = step(k, x, p0, p1);
        p0 = p1;
        p1 = q;
        guard(p0, p1);
        cnt += (unsigned)(__double2hiint(p0) ^ __double2hiint(p1)) >> 31;
      }
    };
    int k = 1;
    for (; k + MC_NB <= n; k += MC_NB) {
      double q[MC_NB];
      int least = 0x7ff00000;
      unsigned c = 0;
      int s = __double2hiint(p1);
#pragma unroll
      for (int u = 0; u < MC_NB; ++u) {
        q[u] = step(k + u, x, u < 2 ? (u == 0 ? p0 : p1) : q[u - 2], u == 0 ? p1 : q[u - 1]);
        const int h = __double2hiint(q[u]);
        least = min(least, h & 0x7fffffff);
        c += (unsigned)(s ^ h) >> 31;
        s = h;
      }
      if (least >= (1023 - MC_LIM) << 20) {
        cnt += c;
        p0 = q[MC_NB - 2];
        p1 = q[MC_NB - 1];
        rescale(p0, p1);
      } else {
        rows(k, k + MC_NB);
      }
    }
    rows(k, n);
    return (int)cnt;
  }
};

__device__ __forceinline__ int sturm_count32(const float *d, const float *e2, int n, float x, float pivmin) {
  float q = d[0] - x;
  if (fabsf(q) <= pivmin) q = -pivmin;
  int c = q < 0.0f;
  for (int k = 1; k < n; ++k) {
    q = d[k] - __fdividef(e2[k - 1], q) - x;
    if (fabsf(q) <= pivmin) q = -pivmin;
    c += q < 0.0f;
  }
  return c;
}

// Sturm count in double-float: q_k = (d_k - x) - e2_{k-1} / q_{k-1} with
// d, e2 and x as hi + lo float pairs.  The quotient is a float estimate
// corrected once by its exact remainder (TwoProd by FMA), about 44 bits; the
// count is then exact for a tridiagonal perturbed by a few 2^-44 relative in
// each entry, the double-float analogue of the FP64 count's backward error.
__device__ __forceinline__ int sturm_count_df(const float *dh, const float *dl, const float *eh, const float *el,
                                              int n, df x, float pivmin) {
  float qh, ql;
  {
    float s, e;
    two_sum(dh[0], -x.hi, s, e);
    e = __fadd_rn(e, __fsub_rn(dl[0], x.lo));
    fast_two_sum(s, e, qh, ql);
  }
  if (fabsf(qh) <= pivmin) {
    qh = -pivmin;
    ql = 0.0f;
  }
  int c = qh < 0.0f;
  for (int k = 1; k < n; ++k) {
    // t = e2 / q
    const float a = eh[k - 1], al = el[k - 1];
    const float th = __fdividef(a, qh);
    const float p = __fmul_rn(th, qh);
    const float pe = __fmaf_rn(th, qh, -p);
    float rem = __fsub_rn(a, p);
    rem = __fsub_rn(rem, pe);
    rem = __fadd_rn(rem, al);
    rem = __fmaf_rn(-th, ql, rem);
    const float tl = __fdividef(rem, qh);
    // q = (d - x) - t as a three-term sum with one renormalisation
    float s1, e1, s2, e2;
    two_sum(dh[k], -x.hi, s1, e1);
    two_sum(s1, -th, s2, e2);
    const float lo = __fadd_rn(__fadd_rn(e1, e2), __fsub_rn(__fsub_rn(dl[k], x.lo), tl));
    fast_two_sum(s2, lo, qh, ql);
    if (fabsf(qh) <= pivmin) {
      qh = -pivmin;
      ql = 0.0f;
    }
    c += qh < 0.0f;
  }
  return c;
}

// One thread per wanted eigenvalue: bisection on Sturm counts of the
// tridiagonal scaled by a power of two to norm 1/2 .. 1.  mode 0: FP64 counts
// from global memory; mode 1 (FP64 form): the tridiagonal in shared memory, the
// interval first narrowed with FP32 Sturm counts, then widened by a margin far
// above the FP32 backward error of the count (64 eps32 (||T|| + |x|)), checked
// with two counts (falling back to the Gerschgorin interval if the check
// fails) and finished in FP64; mode 2 (mixed form): as mode 1 but checked and
// finished with double-float counts, whose accuracy floor (a few 2^-44 ||T||)
// ends the bisection.
__global__ void __launch_bounds__(128) k_bisect(const double *dd, const double *ee, int64_t sd, const int *nvec,
                                                const int64_t *rng, const double *tinfo, double abstol, double *wout,
                                                int64_t *info, int mode) {
  extern __shared__ __align__(16) unsigned char bs_smem[];
  const int b = blockIdx.y;
  const int n = nvec[b];
  const double *d = dd + b * sd;
  const double *e = ee + b * sd;
  const double tnorm = tinfo[b * 8 + 2];
  const int64_t lo_idx = rng[b * 8 + 0];
  const int64_t m = rng[b * 8 + 2];
  if ((int64_t)blockIdx.x * blockDim.x >= m) return;
  // shared memory: (d, e^2) in FP64 (mode 1); then d.hi, e^2.hi (modes 1, 2), d.lo, e^2.lo (mode 2) in float
  double2 *td = (double2 *)bs_smem;
  float *gdh = (float *)(mode == 1 ? (void *)(td + n) : (void *)bs_smem), *ge2h = gdh + n, *gdl = ge2h + n, *ge2l = gdl + n;
  // power of two with sc ||T|| in [1/2, 1); mode 2 keeps the caller's units
  int te = 0;
  if (mode != 2) frexp(tnorm, &te);
  te = max(min(te, 1000), -1000);
  const double sc = ldexp(1.0, -te), isc = ldexp(1.0, te);
  if (mode != 0) {
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
      const double es = (k < n - 1) ? e[k] * sc : 0.0, ds = d[k] * sc, e2 = es * es;
      if (mode == 1) {
        td[k] = make_double2(ds, e2);
        gdh[k] = (float)ds;
        ge2h[k] = (float)e2;
      } else {
        const df dk = df_from(ds), ek = df_from(e2);
        gdh[k] = dk.hi;
        gdl[k] = dk.lo;
        ge2h[k] = ek.hi;
        ge2l[k] = ek.lo;
      }
    }
    __syncthreads();
  }
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  if (tnorm == 0.0) {  // the zero matrix
    wout[b * sd + j] = 0.0;
    return;
  }
  const int64_t idx = lo_idx + j;
  // everything below in units of 1 / sc
  const double gl = tinfo[b * 8 + 0] * sc, gu = tinfo[b * 8 + 1] * sc, tn = tnorm * sc;
  const double pivmin = tinfo[b * 8 + 3] * sc, atol = abstol * sc;
  double lo = gl, hi = gu;
  const double ulp = DBL_EPSILON;
  const float piv32 = fmaxf(1e-30f, (float)pivmin);
  const MinorCount minors{mode == 1 ? td : nullptr, d, e, sc};
  auto count64 = [&](double x) -> int {
    return mode == 2 ? sturm_count_df(gdh, gdl, ge2h, ge2l, n, df_from(x), piv32) : minors(n, x);
  };
  if (mode != 0 && tnorm < 1e30) {
    float lo32 = (float)lo, hi32 = (float)hi;
    const float stop = 16.0f * FLT_EPSILON * (float)tn;
    for (int it = 0; it < 48 && hi32 - lo32 > stop; ++it) {
      const float mid = 0.5f * (lo32 + hi32);
      if (sturm_count32(gdh, ge2h, n, mid, piv32) >= idx)
        hi32 = mid;
      else
        lo32 = mid;
    }
    const double marg = 64.0 * FLT_EPSILON * (tn + fmax(fabs((double)lo32), fabs((double)hi32)));
    const double l2 = fmax(gl, (double)lo32 - marg), h2 = fmin(gu, (double)hi32 + marg);
    if (count64(l2) < idx && count64(h2) >= idx) {
      lo = l2;
      hi = h2;
    }
  }
  // accuracy floor of the double-float count (mode 2)
  const double floor_df = (mode == 2) ? 4.0 * 0x1p-44 * tn : 0.0;
  bool conv = false;
  for (int it = 0; it < 256; ++it) {
    double tol = fmax(fmax(fmax(atol, pivmin), 2.0 * ulp * fmax(fabs(lo), fabs(hi))), floor_df);
    if (hi - lo <= tol) {
      conv = true;
      break;
    }
    double mid = 0.5 * (lo + hi);
    if (count64(mid) >= idx)
      hi = mid;
    else
      lo = mid;
  }
  if (!conv) atomicOr((unsigned long long *)&info[b], (unsigned long long)PP_INFO_NOCONV);
  wout[b * sd + j] = 0.5 * (lo + hi) * isc;
}

// Opt the bisection kernel into the dynamic shared memory it needs for order
// n (done once per size outside any stream capture).
size_t bisect_smem(int64_t n, int mixed) {
  const size_t b = (size_t)n * (mixed ? 4 * sizeof(float) : sizeof(double2) + 2 * sizeof(float));
  return b <= 200 * 1024 ? b : 0;
}

// The attribute applies to the current device only: a high-water mark is
// kept per device.
cudaError_t prepare_bisect(size_t bytes) {
  static std::mutex mu;
  static int done[PP_MAX_DEVICES] = {};
  const int need = (int)bytes;
  if (need > 200 * 1024) return cudaSuccess;
  const int dev = device_index();
  std::lock_guard<std::mutex> g(mu);
  if (dev >= 0 && need <= done[dev]) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_bisect, cudaFuncAttributeMaxDynamicSharedMemorySize, need);
  if (e == cudaSuccess && dev >= 0) done[dev] = need;
  return e;
}

cudaError_t tridiag_eigenvalues(EigWork &w, char range, double vl, double vu, int64_t il, int64_t iu, double abstol,
                                cudaStream_t s, int mixed) {
  const int64_t sd = w.nmax;
  k_tdprep<<<w.B, TD_NT, 0, s>>>(w.d, w.e, sd, w.nvec, range, vl, vu, il, iu, w.rng, w.tinfo, w.info, w.tcErr);
  const size_t smem = bisect_smem(w.nmax, mixed);
  int mode = 0;
  if (smem) {
    mode = mixed ? 2 : 1;
    PP_CUDA_TRY(prepare_bisect(smem));
  }
  // 128 threads a block, or fewer while that leaves SMs idle (a thread's
  // bisection is one dependent chain, so few eigenvalues want many SMs)
  const int mmax = range == 'I' ? (int)(iu - il + 1) : w.nmax;
  int nt = 128;
  while (nt > 32 && cdiv(mmax, nt) * (int64_t)w.B < device_sms()) nt /= 2;
  dim3 g(cdiv(mmax, nt), w.B);
  PP_KT(KT_BISECT, s, (k_bisect<<<g, nt, smem, s>>>(w.d, w.e, sd, w.nvec, w.rng, w.tinfo, abstol, w.w, w.info, mode)));
  count_launch(2);
  return cudaGetLastError();
}


// ===========================================================================
// Stage 3: eigenvectors of T by inverse iteration
// ===========================================================================
// Clusters of consecutive eigenvalues closer than rel * ||T||.
constexpr int CL_NT = 256;
__global__ void __launch_bounds__(CL_NT) k_clusters(const double *ww, int64_t sd, const int64_t *rng, const double *tinfo,
                                                    int *cls, int64_t scl, int *ncl, double rel) {
  __shared__ int wsum[CL_NT / 32];
  const int b = blockIdx.x;
  const int64_t m = rng[b * 8 + 2];
  const double ortol = rel * tinfo[b * 8 + 2];
  const double *w = ww + b * sd;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int c = 0;  // cluster starts before this stretch of CL_NT eigenvalues
  for (int64_t j0 = 0; j0 < m; j0 += CL_NT) {
    const int64_t j = j0 + threadIdx.x;
    const bool start = j < m && (j == 0 || w[j] - w[j - 1] > ortol);
    const unsigned bits = __ballot_sync(0xffffffffu, start);
    if (lane == 0) wsum[warp] = __popc(bits);
    __syncthreads();
    int before = c + __popc(bits & ((1u << lane) - 1u)), all = 0;
    for (int k = 0; k < CL_NT / 32; ++k) {
      if (k < warp) before += wsum[k];
      all += wsum[k];
    }
    if (start) cls[b * scl + before] = (int)j;
    c += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    cls[b * scl + c] = (int)m;
    ncl[b] = c;
  }
}

// Inverse iteration orthogonalises only inside tight clusters (where the
// iterates would otherwise converge to the same vector); eigenvectors of
// eigenvalues further apart but closer than 1e-5 ||T|| keep an overlap of
// about eps ||T|| / gap.  Modified Gram-Schmidt inside those loose clusters
// removes it, one block per cluster (block-wide dot products in FP64).
constexpr int RO_BLOCKS = 64;  // blocks per matrix of k_reorth (cluster c goes to block c mod 64)
template <class R>
__global__ void __launch_bounds__(256) k_reorth(C<R> *Eb, int64_t lde, int64_t sE, const int *nvec, const int *cls,
                                                int64_t scl, const int *ncl) {
  __shared__ double red[32];
  const int b = blockIdx.y;
  const int n = nvec[b];
  C<R> *E = Eb + b * sE;
  const int nc = ncl[b];
  for (int c = blockIdx.x; c < nc; c += gridDim.x) {  // clusters are independent
    const int j0 = cls[b * scl + c], j1 = cls[b * scl + c + 1];
    if (j1 - j0 < 2) continue;
    for (int j = j0 + 1; j < j1; ++j) {
      for (int jp = j0; jp < j; ++jp) {
        double part = 0.0;
        for (int k = threadIdx.x; k < n; k += blockDim.x) part += RT<R>::to(E[k + lde * jp].re) * RT<R>::to(E[k + lde * j].re);
        const double dot = block_sum<256>(part, red);
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
          const double v = RT<R>::to(E[k + lde * j].re) - dot * RT<R>::to(E[k + lde * jp].re);
          E[k + lde * j].re = RT<R>::from(v);
        }
        __syncthreads();
      }
      double part = 0.0;
      for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const double v = RT<R>::to(E[k + lde * j].re);
        part += v * v;
      }
      const double inv = 1.0 / sqrt(block_sum<256>(part, red));
      for (int k = threadIdx.x; k < n; k += blockDim.x)
        E[k + lde * j].re = RT<R>::from(RT<R>::to(E[k + lde * j].re) * inv);
      __syncthreads();
    }
  }
}

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352dU;
  x ^= x >> 15;
  x *= 0x846ca68bU;
  x ^= x >> 16;
  return x;
}

// One thread per cluster of eigenvalues (clusters cbase .. cbase+T-1).
// LU of T - lam I with partial pivoting: row k of U holds 1/u0, u1 and u2 (u2 =
// e(k+1) after a row interchange, else 0) at columns (k, k+1, k+2); l is the
// multiplier, piv marks an interchange.  The factors and the working vector x
// live in scratch, a block's rows in one piece ([row][field][thread]: a warp's
// accesses coalesce and have constant offsets in an unrolled loop); the
// finished vector is written to its column of E once.
// Bound by latency and the instructions of one warp: everything is a recurrence
// over the rows, at 64-85 cycles per dependent FP64 operation (and 16 cycles of
// the SM's FP64 pipe per warp, so a block is one warp).  Hence five passes over
// the rows -- the first right-hand side is eliminated along with the matrix,
// norm and largest component are taken in the U solve, the scaling goes with
// the next pass -- one multiply-add per row on the U solve's chain, reciprocals
// instead of divisions, and each pass requests IV_CH rows ahead of those it
// works on.  n = 2604, all vectors of 4 matrices, with the reorthogonalisation:
// 12.5 ms before (two launches: 2048 threads at most, twelve passes), 4.6 ms
// now; chunks of 8 rows 5.4 ms (registers); the rows of all threads
// interleaved, whose addresses took most of 430 instructions per row, 7.5 ms.
constexpr int IV_CH = 4;  // rows per chunk
constexpr int IV_NT = 32;
template <class R>
__global__ void __launch_bounds__(IV_NT) k_invit(const double *__restrict__ dd, const double *__restrict__ ee, int64_t sd,
                                                 const int *nvec, const double *ww, const int64_t *rng,
                                                 const double *tinfo, const int *cls, int64_t scl, const int *ncl,
                                                 int cbase, int nmax, C<R> *Eb, int64_t lde, int64_t sE, double *scratch,
                                                 uint8_t *pivb, int64_t sS, int64_t sPv, int64_t *info) {
  const int b = blockIdx.y;
  const int c = cbase + blockIdx.x * IV_NT + threadIdx.x;
  if (c >= ncl[b]) return;
  const int n = nvec[b];
  const double *__restrict__ d = dd + b * sd;
  const double *__restrict__ e = ee + b * sd;
  const double *w = ww + b * sd;
  C<R> *E = Eb + b * sE;
  double *S = scratch + b * sS + (int64_t)blockIdx.x * nmax * (IV_F * IV_NT) + threadIdx.x;
  uint8_t *PV = pivb + b * sPv + (int64_t)blockIdx.x * nmax * IV_NT + threadIdx.x;
#define SR0(k) S[(int64_t)(k) * (IV_F * IV_NT)]
#define SU1(k) S[(int64_t)(k) * (IV_F * IV_NT) + IV_NT]
#define SL(k) S[(int64_t)(k) * (IV_F * IV_NT) + 2 * IV_NT]
#define XS(k) S[(int64_t)(k) * (IV_F * IV_NT) + 3 * IV_NT]
#define PIV(k) PV[(int64_t)(k) * IV_NT]
  const double tnorm = tinfo[b * 8 + 2];
  const double eps = DBL_EPSILON * 0.5;
  const double pivtol = fmax(eps * tnorm, DBL_MIN);
  const int j0 = cls[b * scl + c], j1 = cls[b * scl + c + 1];
  const int iters = (j1 - j0 > 1) ? 3 : 2;
  double lam_prev = 0.0;
  int bad = 0;
  struct Row {
    double x, a, u;
    uint8_t pv;
  };
  // rows 0, 1, ... of a pass in chunks, the next chunk's loads ahead of this one's work
  auto pass = [](int rows, auto load, auto work) {
    Row qa[IV_CH], qb[IV_CH];
    auto load_chunk = [&](Row(&q)[IV_CH], int kb) {
#pragma unroll
      for (int u = 0; u < IV_CH; ++u) load(q[u], kb + u);
    };
    auto work_chunk = [&](Row(&q)[IV_CH], int kb) {
#pragma unroll
      for (int u = 0; u < IV_CH; ++u) work(q[u], kb + u);
    };
    const int full = rows / IV_CH * IV_CH;
    if (full > 0) load_chunk(qa, 0);
#pragma unroll 1
    for (int kb = 0; kb < full; kb += 2 * IV_CH) {
      if (kb + IV_CH < full) load_chunk(qb, kb + IV_CH);
      work_chunk(qa, kb);
      if (kb + IV_CH >= full) break;
      if (kb + 2 * IV_CH < full) load_chunk(qa, kb + 2 * IV_CH);
      work_chunk(qb, kb + IV_CH);
    }
#pragma unroll 1
    for (int k = full; k < rows; ++k) {
      load(qa[0], k);
      work(qa[0], k);
    }
  };
  for (int j = j0; j < j1; ++j) {
    double lam = w[j];
    if (j > j0) {
      const double pert = 10.0 * eps * fmax(fabs(lam), 1e-3 * tnorm);
      if (lam <= lam_prev + pert) lam = lam_prev + pert;
    }
    lam_prev = lam;
    // deterministic start vector in (-1, 1), seeded by the eigenvalue index
    // only: results do not depend on the batch slot.  (1 + 24 bits 2^-24 by its
    // bits, to (-1, 1))
    const uint32_t seed = hash32((uint32_t)j * 2654435761u ^ 0x9e3779b9u);
    auto start = [&](int k) {
      const uint32_t h = hash32(seed + (uint32_t)k * 0x85ebca6bu);
      return fma(__hiloint2double(0x3ff00000 | (int)(h >> 12), (int)((h & 0xf00u) << 20)), 2.0, -3.0);
    };
    // ---- factor T - lam I, and L x = (start vector) with the interchanges
    double p = d[0] - lam, qv = (n > 1) ? e[0] : 0.0, ck = qv, xk = start(0);
    pass(
        n - 1,
        [&](Row &q, int k) {
          q.x = e[k + 1];  // (row n - 2: not part of T)
          q.a = d[k + 1];
        },
        [&](const Row &q, int k) {
          const double bk = k + 1 < n - 1 ? q.x : 0.0, ak1 = q.a - lam;
          const double x1 = start(k + 1);
          const bool sw = !(fabs(p) >= fabs(ck));
          const double u0 = sw ? ck : p, r0 = u0 == 0.0 ? 0.0 : recip(u0);
          const double l = (sw ? p : ck) * r0;
          SR0(k) = (fabs(u0) < pivtol) ? 1.0 / copysign(pivtol, u0) : r0;  // 1 / guarded pivot
          SU1(k) = sw ? ak1 : qv;
          SL(k) = l;
          PIV(k) = sw;
          p = sw ? fma(-l, ak1, qv) : fma(-l, qv, ak1);
          qv = sw ? -l * bk : bk;
          XS(k) = sw ? x1 : xk;
          xk = sw ? fma(-l, x1, xk) : fma(-l, xk, x1);
          ck = bk;
        });
    const double rlast = 1.0 / ((fabs(p) < pivtol) ? copysign(pivtol, p) : p);
    bool ok = true, neg = false;
    double sc = 1.0;  // the vector is sc x
#pragma unroll 1
    for (int it = 0; it < iters && ok; ++it) {
      if (it > 0) {  // L solve
        xk = XS(0) * sc;
        pass(
            n - 1,
            [&](Row &q, int k) {
              q.x = XS(k + 1);
              q.a = SL(k);
              q.pv = PIV(k);
            },
            [&](const Row &q, int k) {
              const double x1 = q.x * sc;
              XS(k) = q.pv ? x1 : xk;
              xk = q.pv ? fma(-q.a, x1, xk) : fma(-q.a, xk, x1);
            });
      }
      // U solve from the last row up: y = x/u0 - (u1/u0) y1 - (u2/u0) y2, its
      // squares and its largest component (by its bits; the first of equals)
      double y1 = xk * rlast, y2 = 0.0, nrm2 = y1 * y1;
      long long big = __double_as_longlong(fabs(y1));
      neg = y1 < 0.0;
      XS(n - 1) = y1;
      pass(
          n - 1,
          [&](Row &q, int i) {
            const int k = n - 2 - i;
            q.x = XS(k);
            q.a = SR0(k);
            q.u = SU1(k);
            q.pv = PIV(k);
          },
          [&](const Row &q, int i) {
            const int k = n - 2 - i;
            const double u2 = q.pv && i > 0 ? e[k + 1] : 0.0;
            const double y = fma(-(q.u * q.a), y1, fma(-(u2 * q.a), y2, q.x * q.a));
            XS(k) = y;
            nrm2 = fma(y, y, nrm2);
            const long long m = __double_as_longlong(fabs(y));
            if (m >= big) {
              big = m;
              neg = __double2hiint(y) < 0;
            }
            y2 = y1;
            y1 = y;
          });
      const double amax = __longlong_as_double(big);
      if (!(amax > 0.0) || !isfinite(amax)) {
        ok = false;
        break;
      }
      const double inv = 1.0 / amax;
      // modified Gram-Schmidt against the earlier members of the cluster
      for (int rep = 0; rep < 2 && j > j0; ++rep) {
        for (int jp = j0; jp < j; ++jp) {
          double dot = 0.0;
          auto load = [&](Row &q, int k) {
            q.a = RT<R>::to(E[k + lde * jp].re);
            q.x = XS(k);
          };
          pass(n, load, [&](const Row &q, int) { dot += q.a * q.x; });
          pass(n, load, [&](const Row &q, int k) { XS(k) = q.x - dot * q.a; });
        }
      }
      sc = 1.0;
      if (j > j0 || !(nrm2 > 1e-280 && nrm2 < 1e280)) {
        // the norm of what is left, scaled (or of squares out of range)
        sc = inv;
        nrm2 = 0.0;
        double left = -1.0;
        pass(
            n, [&](Row &q, int k) { q.x = XS(k); },
            [&](const Row &q, int) {
              const double v = q.x * inv;
              nrm2 += v * v;
              if (fabs(v) > left) {
                left = fabs(v);
                neg = v < 0.0;
              }
            });
        if (!(nrm2 > 1e-280)) {
          ok = false;
          break;
        }
      }
      sc = sc / sqrt(nrm2);
    }
    if (!ok) bad = 1;
    // sign convention of dstein: the largest component is positive
    const double ws = neg ? -sc : sc;
    C<R> *Ej = E + lde * j;
    pass(
        n, [&](Row &q, int k) { q.x = XS(k); },
        [&](const Row &q, int k) { Ej[k] = cfrom64<R>(q.x * ws, 0.0); });
  }
  if (bad) atomicOr((unsigned long long *)&info[b], (unsigned long long)PP_INFO_NOORTH);
#undef SR0
#undef SU1
#undef SL
#undef XS
#undef PIV
}

// Threads of k_invit with scratch for an eigenvector each, out of mcap: 2048, or
// all (up to 6144: beyond, the reduction takes seconds) in batches of up to IV_BUSY
// threads.  A thread's time is that of the whole recurrence, so while a launch
// leaves the FP64 pipes idle a second one for the rest costs as much as the first:
// n = 2604, 4 matrices 8.8 -> 4.6 ms, n = 4764, 8 matrices 50 -> 37 ms (969 instead
// of 983 ms a pass).  Past that the pipes are busy either way and the scratch (33 n
// bytes a thread) is not worth it: n = 4764, 24 matrices 53 -> 38 ms of a pass of
// 2696 and 2699 ms for 10 GB more, n = 2604, 48 matrices 26 -> 27 ms for 3 GB.
constexpr int64_t IV_BUSY = 40960;
int64_t invit_threads(int64_t mcap, int B) {
  const int64_t all = std::min<int64_t>((mcap + 63) / 64 * 64, 6144);
  return B > 0 && all * B <= IV_BUSY ? all : std::min<int64_t>(all, 2048);
}

template <class R>
cudaError_t tridiag_eigenvectors(EigWork &w, cudaStream_t s) {
  const int64_t sd = w.nmax;
  const int64_t scl = w.nmax + 1;
  k_clusters<<<w.B, CL_NT, 0, s>>>(w.w, sd, w.rng, w.tinfo, w.cls, scl, w.ncl, 1e-7);
  count_launch(1);
  const int64_t T = w.scratch_threads;
  const int64_t sS = (int64_t)IV_F * w.nmax * T;
  const int64_t sPv = (int64_t)w.nmax * T;
  for (int64_t cb = 0; cb < w.mcap; cb += T) {
    dim3 g(cdiv(std::min<int64_t>(T, w.mcap - cb), IV_NT), w.B);
    PP_KT(KT_INVIT, s, (k_invit<R><<<g, IV_NT, 0, s>>>(w.d, w.e, sd, w.nvec, w.w, w.rng, w.tinfo, w.cls, scl, w.ncl,
                                                    (int)cb, w.nmax, (C<R> *)w.E, w.lde, w.sE, w.scratch, w.piv, sS,
                                                    sPv, w.info)));
    count_launch(1);
  }
  k_clusters<<<w.B, CL_NT, 0, s>>>(w.w, sd, w.rng, w.tinfo, w.cls, scl, w.ncl, 1e-5);
  PP_KT(KT_INVIT, s, (k_reorth<R><<<dim3(RO_BLOCKS, w.B), 256, 0, s>>>((C<R> *)w.E, w.lde, w.sE, w.nvec, w.cls, scl, w.ncl)));
  count_launch(2);
  return cudaGetLastError();
}

// ===========================================================================
// Stage 4: back-transform E = Q Z
// ===========================================================================
constexpr int BT_J = 32;     // columns per block
constexpr int BT_NT = 128;   // threads: a column and 8 of the 32 panel columns each
constexpr int BT_RK = 16;    // rows per k-step
// Rows per split-K chunk of `rows`: 8 chunks, 32 to 256 rows.  (64 columns and
// 512 rows per block left half of the SMs without work: 4 matrices of order
// 1092 with 1092 columns 935 us -> 606 us per panel.)
constexpr int BT_CHUNKS = 8, BT_RMIN = 32, BT_RMAX = 256;
static int bt_chunk(int rows) { return std::max(BT_RMIN, std::min(BT_RMAX, cdiv(cdiv(rows, BT_CHUNKS), BT_RK) * BT_RK)); }

// Wp[ks][a][j] = sum_{r in chunk ks} conj(V(r,a)) X(r,j) for a < jb.
// V(r,a) = A(r, k0+a) for r >= k0+a+1 (zero above); j < the matrix's m, or
// ncol_fixed.
template <class R>
__global__ void __launch_bounds__(BT_NT) k_vhx(const C<R> *Ab, int64_t lda, int64_t sA, const C<R> *Xb, int64_t ldx,
                                             int64_t sX, const int *nvec, const int64_t *rng, int k0, int jb,
                                             C<R> *Wp, int64_t ldwp, int64_t sWp, int ncol_fixed, int rch) {
  __shared__ C<R> sV[BT_RK][32];
  __shared__ C<R> sXt[BT_RK][BT_J];
  const int b = blockIdx.z;
  const int n = nvec[b];
  const int ncol = ncol_fixed > 0 ? ncol_fixed : (int)rng[b * 8 + 2];
  const int j0 = blockIdx.x * BT_J;
  const int ks = blockIdx.y;
  const int rbeg = k0 + 1 + ks * rch;
  if (j0 >= ncol || rbeg >= n) return;
  const C<R> *A = Ab + b * sA;
  const C<R> *X = Xb + b * sX;
  const int64_t ldX = ldx;
  const int tj = threadIdx.x & 31, ta = threadIdx.x >> 5;
  C<R> acc[8];
#pragma unroll
  for (int p = 0; p < 8; ++p) acc[p] = cz<R>();
  const int rend = min(n, rbeg + rch);
  for (int r0 = rbeg; r0 < rend; r0 += BT_RK) {
    for (int e = threadIdx.x; e < BT_RK * 32; e += BT_NT) {
      const int a = e & 31, rr = e >> 5;
      const int r = r0 + rr;
      sV[rr][a] = (a < jb && r < rend && r >= k0 + a + 1) ? cconj(A[r + lda * (k0 + a)]) : cz<R>();
    }
    for (int e = threadIdx.x; e < BT_RK * BT_J; e += BT_NT) {
      const int jx = e & 31, rr = e >> 5;
      const int r = r0 + rr, j = j0 + jx;
      const bool ok = r < rend && j < ncol;
      sXt[rr][jx] = ok ? X[r + ldX * j] : cz<R>();
    }
    __syncthreads();
#pragma unroll 4
    for (int rr = 0; rr < BT_RK; ++rr) {
      const C<R> xv = sXt[rr][tj];
#pragma unroll
      for (int p = 0; p < 8; ++p) cmac(acc[p], sV[rr][ta + 4 * p], xv);
    }
    __syncthreads();
  }
  const int j = j0 + tj;
  if (j < ncol) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const int a = ta + 4 * p;
      if (a < jb) Wp[b * sWp + ((int64_t)ks * 32 + a) * ldwp + j] = cfin(acc[p]);
    }
  }
}

// Sum the split-K partials of V^H X and apply the panel's compact-WY factor
// (Tf at Tf + 1024 b, upper triangular): mode 1 Y = Tf (V^H X), mode 2
// Y = Tf^H (V^H X); written to Wb.
// Block of BR_NT threads = 32 columns j x 8 groups of panel rows a (a = g,
// g + 8, g + 16, g + 24): the partials are summed into shared memory, then
// every thread forms its four rows of the product with Tf.  (Tf is converted to
// R once per block: with the conversion at each use the FP64 pipe bound the
// double-float form: n = 2604, 4 matrices 132 -> 38 us a panel, n = 4764, 8
// matrices 147 -> 51 us.)
constexpr int BR_NT = 256;
template <class R>
__global__ void __launch_bounds__(BR_NT) k_btred(const C<R> *Wp, int64_t ldwp, int64_t sWp, const int *nvec,
                                                 const int64_t *rng, int k0, int jb, int mode, const z64 *Tf,
                                                 C<R> *Wb, int64_t sWb, int ncol_fixed, int rch, int nks_fixed = 0) {
  __shared__ C<R> col[32][33];
  __shared__ C<R> sT[32][33];
  const int b = blockIdx.y;
  const int n = nvec[b];
  const int ncol = ncol_fixed > 0 ? ncol_fixed : (int)rng[b * 8 + 2];
  // split-K partials to sum: one per rch rows, or nks_fixed
  const int nks = nks_fixed > 0 ? (n - k0 - 1 > 0 ? nks_fixed : 0) : (n - k0 - 1 + rch - 1) / rch;
  const int j0 = blockIdx.x * 32;
  if (j0 >= ncol || nks <= 0) return;
  for (int e = threadIdx.x; e < 32 * 32; e += BR_NT) sT[e / 32][e % 32] = cfrom64<R>(Tf[b * 1024 + e]);
  const int jl = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int j = j0 + jl;
  for (int a = g; a < jb; a += 8) {
    C<R> s = cz<R>();
    if (j < ncol)
      for (int ks = 0; ks < nks; ++ks) s = cadd(s, Wp[b * sWp + ((int64_t)ks * 32 + a) * ldwp + j]);
    col[a][jl] = s;
  }
  __syncthreads();
  if (j >= ncol) return;
  for (int a = g; a < jb; a += 8) {
    C<R> acc = cz<R>();
    if (mode == 1) {
      for (int a2 = a; a2 < jb; ++a2) cmac(acc, sT[a][a2], col[a2][jl]);
    } else {  // mode 2: Tf^H (lower triangular)
      for (int a2 = 0; a2 <= a; ++a2) cmac(acc, cconj(sT[a2][a]), col[a2][jl]);
    }
    Wb[b * sWb + (int64_t)a * ldwp + j] = cfin(acc);
  }
}

// Compact-WY factors of every panel in one launch, one block per (panel,
// matrix): the Gram matrix G = V^H V of the panel's Householder vectors
// (products in the arithmetic R, rows staged WY_RK at a time and the sums
// renormalised after each stage, each thread two entries above the diagonal), then Tf by
// zlarft's forward columnwise recurrence in FP64: Tf(a,a) = tau_a,
// Tf(0:a, a) = -tau_a Tf(0:a, 0:a) G(0:a, a).  Tf of panel P for matrix b
// goes to Tf + P sTfp + 1024 b (row-major 32 x 32).  Panel widths follow the
// batch's largest order (nref = nmax - 1); reflectors past a matrix's own
// order have tau = 0 and give zero columns of Tf.
constexpr int WY_RK = 16;
template <class R>
__global__ void __launch_bounds__(256) k_wy_factors(const C<R> *Ab, int64_t lda, int64_t sA, const int *nvec,
                                                     const z64 *tau, int64_t sd, int nb, int nref, z64 *Tf,
                                                     int64_t sTfp) {
  __shared__ C<R> sV[WY_RK][33];
  __shared__ z64 G[32][33];
  __shared__ z64 sT[32][33];
  const int P = blockIdx.x, b = blockIdx.y;
  const int n = nvec[b];
  const int k0 = P * nb;
  const int jb = min(nb, nref - k0);
  const C<R> *A = Ab + b * sA;
  const int tid = threadIdx.x;
  // the 496 entries G(a, j), a < j, that the recurrence reads: two per thread
  int ga[2], gj[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int t = min(tid + 256 * q, 495);
    int j = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)t)) * 0.5f);
    while (j * (j - 1) / 2 > t) --j;
    while (j * (j + 1) / 2 <= t) ++j;
    gj[q] = j;
    ga[q] = t - j * (j - 1) / 2;
  }
  C<R> acc[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) acc[q] = cz<R>();
  for (int r0 = k0 + 1; r0 < n; r0 += WY_RK) {
    for (int e = tid; e < WY_RK * 32; e += 256) {
      const int a = e & 31, rr = e >> 5, r = r0 + rr;
      sV[rr][a] = (a < jb && r < n && r >= k0 + a + 1) ? A[r + lda * (k0 + a)] : cz<R>();
    }
    __syncthreads();
#pragma unroll 4
    for (int rr = 0; rr < WY_RK; ++rr) {
#pragma unroll
      for (int q = 0; q < 2; ++q) cmacc(acc[q], sV[rr][ga[q]], sV[rr][gj[q]]);
    }
    // renormalise after every WY_RK rows: the unnormalised low word of the
    // multiply-add is meant for short sums, the panel runs over all n rows
#pragma unroll
    for (int q = 0; q < 2; ++q) acc[q] = cfin(acc[q]);
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) G[ga[q]][gj[q]] = cto64(cfin(acc[q]));
  for (int e = tid; e < 1024; e += 256) sT[e / 32][e % 32] = z64{0.0, 0.0};
  __syncthreads();
  if (tid < 32) {
    const int a = tid;
    for (int jj = 0; jj < jb; ++jj) {
      const int i = k0 + jj;
      const z64 tj = (i < n - 1) ? tau[b * sd + i] : z64{0.0, 0.0};
      z64 acc2{0.0, 0.0};
      for (int a2 = a; a2 < jj; ++a2) {
        const z64 g = G[a2][jj];
        const z64 tt = sT[a][a2];
        acc2.re += tt.re * g.re - tt.im * g.im;
        acc2.im += tt.re * g.im + tt.im * g.re;
      }
      __syncwarp();
      if (a < jj) {
        const z64 v = zmul(tj, acc2);
        sT[a][jj] = z64{-v.re, -v.im};
      }
      if (a == jj) sT[jj][jj] = tj;
      __syncwarp();
    }
  }
  __syncthreads();
  z64 *T = Tf + (int64_t)P * sTfp + (int64_t)b * 1024;
  for (int e = tid; e < 1024; e += 256) T[e] = sT[e / 32][e % 32];
}

// E(r, j) -= sum_a V(r, a) Y(a, j), r in [k0+1, n), j < m.
constexpr int AV_T = 32, AV_K = 16, AV_P = AV_T / 16;  // (64 x 64 tiles: too few blocks for orders of a few hundred)
template <class R>
__global__ void __launch_bounds__(256) k_applyV(const C<R> *Ab, int64_t lda, int64_t sA, const C<R> *Wb,
                                                int64_t ldwp, int64_t sWb, C<R> *Eb, int64_t lde, int64_t sE,
                                                const int *nvec, const int64_t *rng, int k0, int jb, int ncol_fixed) {
  __shared__ C<R> sV[AV_K][AV_T];
  __shared__ C<R> sY[AV_K][AV_T];
  const int b = blockIdx.z;
  const int n = nvec[b];
  const int m = ncol_fixed > 0 ? ncol_fixed : (int)rng[b * 8 + 2];
  const int r0 = k0 + 1 + blockIdx.x * AV_T, c0 = blockIdx.y * AV_T;
  if (r0 >= n || c0 >= m) return;
  const C<R> *A = Ab + b * sA;
  const C<R> *Y = Wb + b * sWb;
  C<R> *E = Eb + b * sE;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  C<R> acc[AV_P][AV_P];
#pragma unroll
  for (int p = 0; p < AV_P; ++p)
#pragma unroll
    for (int q = 0; q < AV_P; ++q) acc[p][q] = cz<R>();
  for (int kc = 0; kc < jb; kc += AV_K) {
    for (int e = threadIdx.x; e < AV_K * AV_T; e += 256) {
      const int x = e % AV_T, y = e / AV_T;
      const int a = kc + y;
      const int r = r0 + x, c = c0 + x;
      sV[y][x] = (a < jb && r < n && r >= k0 + a + 1) ? A[r + lda * (k0 + a)] : cz<R>();
      sY[y][x] = (a < jb && c < m) ? Y[(int64_t)a * ldwp + c] : cz<R>();
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < AV_K; ++k) {
      C<R> v[AV_P], y[AV_P];
#pragma unroll
      for (int p = 0; p < AV_P; ++p) {
        v[p] = sV[k][tx + 16 * p];
        y[p] = sY[k][ty + 16 * p];
      }
#pragma unroll
      for (int p = 0; p < AV_P; ++p)
#pragma unroll
        for (int q = 0; q < AV_P; ++q) cmac(acc[p][q], v[p], y[q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < AV_P; ++p)
#pragma unroll
    for (int q = 0; q < AV_P; ++q) {
      const int r = r0 + tx + 16 * p, c = c0 + ty + 16 * q;
      if (r < n && c < m) {
        C<R> *x = &E[r + lde * c];
        *x = csub(*x, cfin(acc[p][q]));
      }
    }
}

template <class R>
cudaError_t back_transform(EigWork &w, cudaStream_t s) {
  const int B = w.B, nmax = w.nmax, nb = w.nb;
  if (nmax < 2) return cudaSuccess;
  const int nref = nmax - 1;  // reflector columns 0 .. nmax-2
  const int64_t ldwp = w.ldwp;
  const int64_t sWp = (int64_t)w.ksplit * 32 * ldwp;
  const int64_t sWb = (int64_t)32 * ldwp;
  const int64_t sd = w.nmax;
  C<R> *A = (C<R> *)w.A;
  C<R> *E = (C<R> *)w.E;
  C<R> *Wp = (C<R> *)w.Wp;
  C<R> *Wb = (C<R> *)w.Wb;
  // compact-WY factors of all panels
  PP_KT(KT_BTRED, s, (k_wy_factors<R><<<dim3(cdiv(nref, nb), B), 256, 0, s>>>(A, w.lda, w.sA, w.nvec, w.tau, sd, nb,
                                                                           nref, w.Tf, w.sTfp)));
  count_launch(1);
  const int kstart = ((nref - 1) / nb) * nb;
  for (int k0 = kstart; k0 >= 0; k0 -= nb) {
    const int jb = min(nb, nref - k0);
    const int rch = bt_chunk(nmax - k0 - 1), ks = cdiv(nmax - k0 - 1, rch);
    const z64 *Tf = w.Tf + (int64_t)(k0 / nb) * w.sTfp;
    // Y = Tf V^H E ; E -= V Y (on the tensor cores in the double-float form,
    // over all mcap columns)
    const bool tc = std::is_same<R, df>::value && w.tcS && tc_enabled();
    if (tc) {
      PP_CUDA_TRY(vhx_tc(w, k0, jb, (const zdf *)E, w.lde, w.sE, w.mcap, (zdf *)Wp, ldwp, sWp, s));
      PP_KT(KT_BTRED, s, (k_btred<R><<<dim3(cdiv(w.mcap, 32), B), BR_NT, 0, s>>>(Wp, ldwp, sWp, w.nvec, w.rng, k0, jb, 1, Tf, Wb, sWb, w.mcap, rch, vhx_tc_splits(w))));
      PP_CUDA_TRY(applyV_tc(w, k0, jb, (zdf *)E, w.lde, w.sE, (const zdf *)Wb, ldwp, sWb, w.mcap, s));
      count_launch(1);
    } else {
      PP_KT(KT_VHX, s, (k_vhx<R><<<dim3(cdiv(w.mcap, BT_J), ks, B), BT_NT, 0, s>>>(A, w.lda, w.sA, E, w.lde, w.sE, w.nvec, w.rng, k0,
                                                               jb, Wp, ldwp, sWp, 0, rch)));
      PP_KT(KT_BTRED, s, (k_btred<R><<<dim3(cdiv(w.mcap, 32), B), BR_NT, 0, s>>>(Wp, ldwp, sWp, w.nvec, w.rng, k0, jb, 1, Tf, Wb, sWb, 0, rch)));
      PP_KT(KT_APPLYV, s, (k_applyV<R><<<dim3(cdiv(nmax - k0 - 1, AV_T), cdiv(w.mcap, AV_T), B), 256, 0, s>>>(
          A, w.lda, w.sA, Wb, ldwp, sWb, E, w.lde, w.sE, w.nvec, w.rng, k0, jb, 0)));
      count_launch(3);
    }
  }
  return cudaGetLastError();
}

// X = P^T (unit columns at the selected rows)
template <class R>
__global__ void k_rows_init(C<R> *Xb, int64_t ldx, int64_t sX, const int *rows, int nrows, const int *nvec) {
  const int b = blockIdx.z;
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y;
  if (r >= nvec[b] || k >= nrows) return;
  Xb[b * sX + r + ldx * k] = (r == rows[k]) ? cfrom64<R>(1.0, 0.0) : cz<R>();
}

// Eb(k, j) = sum_r conj(X(r,k)) Z(r,j), Z real (stored as complex with zero
// imaginary part): the selected rows of E = Q Z.
constexpr int XZ_T = 64, XZ_K = 16;
template <class R>
__global__ void __launch_bounds__(256) k_xhz(const C<R> *Xb, int64_t ldx, int64_t sX, const C<R> *Zb, int64_t ldz,
                                             int64_t sZ, C<R> *Eb, int64_t lde, int64_t sE, const int *nvec,
                                             const int64_t *rng, int nrows) {
  __shared__ C<R> sXt[XZ_K][XZ_T];
  __shared__ R sZt[XZ_K][XZ_T];
  const int b = blockIdx.z;
  const int n = nvec[b];
  const int m = (int)rng[b * 8 + 2];
  const int k0 = blockIdx.x * XZ_T, j0 = blockIdx.y * XZ_T;
  if (k0 >= nrows || j0 >= m) return;
  const C<R> *X = Xb + b * sX;
  const C<R> *Z = Zb + b * sZ;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  C<R> acc[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = cz<R>();
  for (int r0 = 0; r0 < n; r0 += XZ_K) {
    for (int e = threadIdx.x; e < XZ_K * XZ_T; e += 256) {
      const int x = e % XZ_T, y = e / XZ_T;
      const int r = r0 + y;
      sXt[y][x] = (r < n && k0 + x < nrows) ? cconj(X[r + ldx * (k0 + x)]) : cz<R>();
      sZt[y][x] = (r < n && j0 + x < m) ? Z[r + ldz * (j0 + x)].re : RT<R>::zero();
    }
    __syncthreads();
#pragma unroll 4
    for (int y = 0; y < XZ_K; ++y) {
      C<R> xv[4];
      R zv[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        xv[p] = sXt[y][tx + 16 * p];
        zv[p] = sZt[y][ty + 16 * p];
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          RT<R>::mac(acc[p][q].re, xv[p].re, zv[q]);
          RT<R>::mac(acc[p][q].im, xv[p].im, zv[q]);
        }
    }
    __syncthreads();
  }
  C<R> *E = Eb + b * sE;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = k0 + tx + 16 * p, j = j0 + ty + 16 * q;
      if (k < nrows && j < m) E[k + lde * j] = cfin(acc[p][q]);
    }
}

template <class R>
cudaError_t back_transform_rows(EigWork &w, const int *d_rows, int nrows, cudaStream_t s) {
  const int B = w.B, nmax = w.nmax, nb = w.nb;
  if (nrows <= 0) return cudaSuccess;
  const int64_t ldx = w.lda, sX = (int64_t)w.lda * w.nbr;
  C<R> *A = (C<R> *)w.A;
  C<R> *X = (C<R> *)w.Xr;
  C<R> *Wp = (C<R> *)w.Wp;
  C<R> *Wb = (C<R> *)w.Wb;
  const int64_t ldwp = w.ldwp;
  const int64_t sWp = (int64_t)w.ksplit * 32 * ldwp;
  const int64_t sWb = (int64_t)32 * ldwp;
  const int64_t sd = w.nmax;
  k_rows_init<R><<<dim3(cdiv(nmax, 256), nrows, B), 256, 0, s>>>(X, ldx, sX, d_rows, nrows, w.nvec);
  count_launch(1);
  // X <- Q^H X = Q_last^H ... Q_0^H X: panels in forward order, Tf^H
  const int nref = nmax - 1;
  PP_KT(KT_BTRED, s, (k_wy_factors<R><<<dim3(cdiv(nref, nb), B), 256, 0, s>>>(A, w.lda, w.sA, w.nvec, w.tau, sd, nb,
                                                                           nref, w.Tf, w.sTfp)));
  count_launch(1);
  for (int k0 = 0; k0 < nref; k0 += nb) {
    const int jb = min(nb, nref - k0);
    const int rch = bt_chunk(nmax - k0 - 1), ks = cdiv(nmax - k0 - 1, rch);
    const z64 *Tf = w.Tf + (int64_t)(k0 / nb) * w.sTfp;
    const bool tc = std::is_same<R, df>::value && w.tcS && tc_enabled();
    if (tc) {
      PP_CUDA_TRY(vhx_tc(w, k0, jb, (const zdf *)X, ldx, sX, nrows, (zdf *)Wp, ldwp, sWp, s));
    } else {
      PP_KT(KT_VHX, s, (k_vhx<R><<<dim3(cdiv(nrows, BT_J), ks, B), BT_NT, 0, s>>>(A, w.lda, w.sA, X, ldx, sX, w.nvec,
                                                                               w.rng, k0, jb, Wp, ldwp, sWp, nrows,
                                                                               rch)));
    }
    PP_KT(KT_BTRED, s, (k_btred<R><<<dim3(cdiv(nrows, 32), B), BR_NT, 0, s>>>(Wp, ldwp, sWp, w.nvec, w.rng, k0, jb, 2,
                                                                          Tf, Wb, sWb, nrows, rch,
                                                                          tc ? vhx_tc_splits(w) : 0)));
    if (tc) {
      PP_CUDA_TRY(applyV_tc(w, k0, jb, (zdf *)X, ldx, sX, (const zdf *)Wb, ldwp, sWb, nrows, s));
    } else {
      PP_KT(KT_APPLYV, s, (k_applyV<R><<<dim3(cdiv(nmax - k0 - 1, AV_T), cdiv(nrows, AV_T), B), 256, 0, s>>>(
                              A, w.lda, w.sA, Wb, ldwp, sWb, X, ldx, sX, w.nvec, w.rng, k0, jb, nrows)));
    }
    count_launch(tc ? 1 : 3);  // the tensor-core helpers count their own launches
  }
  // Eb = X^H Z
  if (std::is_same<R, df>::value && w.tcS && tc_enabled()) {
    PP_CUDA_TRY(xhz_tc(w, (const zdf *)X, ldx, sX, nrows, (const zdf *)w.E, w.lde, w.sE, (zdf *)w.Eb,
                       (int64_t)w.nbr, (int64_t)w.nbr * w.mcap, s));
  } else {
    PP_KT(KT_XHZ, s, (k_xhz<R><<<dim3(cdiv(nrows, XZ_T), cdiv(w.mcap, XZ_T), B), 256, 0, s>>>(
                         X, ldx, sX, (const C<R> *)w.E, w.lde, w.sE, (C<R> *)w.Eb, (int64_t)w.nbr,
                         (int64_t)w.nbr * w.mcap, w.nvec, w.rng, nrows)));
    count_launch(1);
  }
  return cudaGetLastError();
}

// explicit instantiations
template cudaError_t tridiagonalize<double>(EigWork &, cudaStream_t);
template cudaError_t tridiagonalize<df>(EigWork &, cudaStream_t);
template cudaError_t tridiag_eigenvectors<double>(EigWork &, cudaStream_t);
template cudaError_t tridiag_eigenvectors<df>(EigWork &, cudaStream_t);
template cudaError_t back_transform<double>(EigWork &, cudaStream_t);
template cudaError_t back_transform<df>(EigWork &, cudaStream_t);
template cudaError_t back_transform_rows<double>(EigWork &, const int *, int, cudaStream_t);
template cudaError_t back_transform_rows<df>(EigWork &, const int *, int, cudaStream_t);

}  // namespace pp
