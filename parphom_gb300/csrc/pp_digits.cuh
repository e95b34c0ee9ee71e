// Number formats of the tensor-core products: double-float values as digits on a
// fixed-point grid, and sums of digit products as double-float values.
#pragma once
#include <cfloat>
#include <cstdint>
#include <cuda_fp16.h>

#include "pp_common.cuh"

namespace pp {

// 2^e as a float (exact for -126 <= e <= 127)
__device__ __forceinline__ float pow2f(int e) {
  return (e >= -126 && e <= 127) ? __int_as_float((e + 127) << 23) : ldexpf(1.0f, e);
}

// Digits of the long-K operands.  v = x 2^-E, |v| < 1, as the 56-bit integer
// n = rint(2^56 v) plus 512 2^48 and 128 in each of the six lower bytes: those
// bytes less 128 are the digits m_1 .. m_6 and the upper 16 bits less 512 are m_0 in
//   v = sum_{s=0..6} 2^-8(s+1) m_s,  |m_0| <= 256, |m_s| <= 128 for s > 0,
// residual below 2^-57: the grid and the residual of slice_row.  Three exact
// extractions (22, 22 and 12 bits) by adding constants; the bits of the three sums
// are the three integers up to constants.
struct Fixed56 {
  uint32_t lo, hi;
};
__device__ __forceinline__ Fixed56 to_fixed(float hi, float lo) {
  constexpr float M0 = 3.f, M1 = 1.5f * 0x1p-21f, M2 = 1.5f * 0x1p-33f;  // ulps 2^-22, 2^-44, 2^-56
  constexpr uint64_t off = 0x0200808080808080ull - ((uint64_t)0x40400000u << 34) - ((uint64_t)0x35400000u << 12) -
                           0x2f400000u;
  const float t0 = __fadd_rn(hi, M0);
  float r = __fsub_rn(hi, __fsub_rn(t0, M0)), e;
  fast_two_sum(r, lo, r, e);  // |r| >= |lo| or r = 0
  const float t1 = __fadd_rn(r, M1);
  r = __fadd_rn(__fsub_rn(r, __fsub_rn(t1, M1)), e);
  const float t2 = __fadd_rn(r, M2);
  const uint64_t n = (uint64_t)__float_as_uint(t1) * 4096u +
                     (((uint64_t)(__float_as_uint(t0) << 2) << 32) | __float_as_uint(t2)) + off;
  return Fixed56{(uint32_t)n, (uint32_t)(n >> 32)};
}
// digit S of two numbers in half precision (low half: a): 1024 + the digit's
// field by its bits, less 1536 or 1152 (exact).  bf16 has no room for an 8-bit
// byte below its leading bit, and costs five instructions here instead of two
// or three.
template <int S>
__device__ __forceinline__ uint32_t digit2(Fixed56 a, Fixed56 b) {
  constexpr uint32_t k = S <= 2 ? 2 - S : 6 - S;  // byte of the word
  constexpr uint16_t bias = S == 0 ? 0x6600 : 0x6480;
  const uint32_t w = S == 0 ? __byte_perm(a.hi, b.hi, 0x7632)
                            : __byte_perm(S <= 2 ? a.hi : a.lo, S <= 2 ? b.hi : b.lo, (k + 4) << 8 | k) & 0x00ff00ffu;
  const uint32_t x = w | 0x64006400u;
  const __half2 h = __hsub2(*(const __half2 *)&x, __half2{__ushort_as_half(bias), __ushort_as_half(bias)});
  return *(const uint32_t *)&h;
}

// Exponent E of a row's grid from its largest magnitude (its elements are below
// 2^E), and the scaling by 2^-E in up to two exact steps (2^-E exceeds the
// float range for subnormal rows, e.g. the far tail of a localised
// eigenvector).  A row with an infinity or NaN gets an exponent that makes every
// product of it non-finite.
constexpr int LK_NONFINITE = 1 << 20;
__device__ __forceinline__ float max_abs(float m, float x) {  // NaN if one is
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(m), "f"(fabsf(x)));
  return r;
}
__device__ __forceinline__ int grid_exp(float amax) {
  if (!(amax <= FLT_MAX)) return LK_NONFINITE;
  int E = 0;
  if (amax > 0.f) frexpf(amax, &E);
  return E;
}
__device__ __forceinline__ float grid_scale(int E) { return E == LK_NONFINITE ? 0.f : pow2f(E < -100 ? -E - 100 : -E); }
// x[0..N) to grid integers (warp-wide call)
template <int N>
__device__ __forceinline__ void to_fixed(const df *x, int E, bool neg, Fixed56 *f) {
  const float sc = neg ? -grid_scale(E) : grid_scale(E);
  if (__any_sync(0xffffffffu, E < -100)) {
    const float pre = E < -100 ? 0x1p100f : 1.f;
#pragma unroll
    for (int t = 0; t < N; ++t)
      f[t] = to_fixed(__fmul_rn(__fmul_rn(x[t].hi, pre), sc), __fmul_rn(__fmul_rn(x[t].lo, pre), sc));
  } else {
#pragma unroll
    for (int t = 0; t < N; ++t) f[t] = to_fixed(__fmul_rn(x[t].hi, sc), __fmul_rn(x[t].lo, sc));
  }
}

// s += a 2^-8U for one group of the sum over u of a_u 2^-8u, in the order
// u = 6, 5, 4, 0, 1, 2, 3.  The a_u are integers of at most 2^24 in magnitude.
// Groups 4-6 add up in float (rounding error below 2^-32 of the unit of group
// 0).  In groups 1-3 s.hi is a multiple of 2^-8(U-1) and so of ulp(a 2^-8U),
// which makes the three-operation sum exact without an ordering by magnitude.
template <int U>
__device__ __forceinline__ void fold_group(df &s, float a) {
  constexpr float w = 1.f / (float)((uint64_t)1 << (8 * U));
  if (U == 6)
    s.lo = __fmul_rn(a, w);
  else if (U >= 4)
    s.lo = __fmaf_rn(a, w, s.lo);
  else if (U == 0)
    s.hi = a;
  else {
    const float h = __fmaf_rn(a, w, s.hi);
    s.lo = __fadd_rn(s.lo, __fmaf_rn(a, w, __fsub_rn(s.hi, h)));
    s.hi = h;
  }
}
__device__ __forceinline__ df fold_done(df s) {
  df r;
  two_sum(s.hi, s.lo, r.hi, r.lo);
  return r;
}
// s += a 2^-8U in the order 6, 5, ..., 0 (see fold_group): here s.hi is a
// multiple of 2^-8(U+1) below 2^(24-8(U+1)), so that a 2^-8U is a multiple of
// ulp(s.hi) and the three-operation sum is exact as well.
template <int U>
__device__ __forceinline__ void fold_up(df &s, float a) {
  constexpr float w = 1.f / (float)((uint64_t)1 << (8 * U));
  if (U == 6)
    s.lo = __fmul_rn(a, w);
  else if (U >= 4)
    s.lo = __fmaf_rn(a, w, s.lo);
  else if (U == 3)
    s.hi = __fmul_rn(a, w);
  else {
    const float h = __fmaf_rn(a, w, s.hi);
    s.lo = __fadd_rn(s.lo, __fsub_rn(s.hi, __fmaf_rn(a, -w, h)));
    s.hi = h;
  }
}

}  // namespace pp
