// Sums that have to keep more than the terms' own precision, and a reciprocal.
#pragma once
#include "pp_common.cuh"

namespace pp {

// Sums over threads.  Double: plain FP64 adds.  Double-float: an unevaluated
// sum of three floats, whose additions lose nothing above ~2^-70 of the
// largest term -- no less than an FP64 sum, without the FP64 pipe (a
// dependent FP64 add waits 64-150 cycles on this chip, and a division or a
// square root 560-690; such chains were most of a column's time).
struct tf {
  float a, b, c;
};
template <class R>
struct Sum;
template <>
struct Sum<double> {
  typedef double T;
  PP_D static T zero() { return 0.0; }
  PP_D static T from(double x) { return x; }
  PP_D static T add(T x, T y) { return x + y; }
  PP_D static T sub(T x, T y) { return x - y; }
  PP_D static T mul(double x, double y) { return x * y; }
  PP_D static T mul2(double x, double y, double u, double v) { return fma(u, v, x * y); }  // x y + u v
  PP_D static T shfl_xor(T x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); }
  PP_D static double to(T x) { return x; }
  PP_D static double toR(T x) { return x; }
};
template <>
struct Sum<df> {
  typedef tf T;
  PP_D static T zero() { return tf{0.f, 0.f, 0.f}; }
  PP_D static T from(df x) { return tf{x.hi, x.lo, 0.f}; }
  PP_D static T add(T x, T y) {
    float s, e0, t, e1, u, e2;
    two_sum(x.a, y.a, s, e0);
    two_sum(x.b, y.b, t, e1);
    two_sum(t, e0, u, e2);
    return tf{s, u, __fadd_rn(__fadd_rn(x.c, y.c), __fadd_rn(e1, e2))};
  }
  PP_D static T sub(T x, T y) { return add(x, tf{-y.a, -y.b, -y.c}); }
  // the product of two double-floats with every partial product kept
  PP_D static T mul(df x, df y) {
    const float p = __fmul_rn(x.hi, y.hi), pe = __fmaf_rn(x.hi, y.hi, -p);
    const float q = __fmul_rn(x.hi, y.lo), qe = __fmaf_rn(x.hi, y.lo, -q);
    const float r = __fmul_rn(x.lo, y.hi), re = __fmaf_rn(x.lo, y.hi, -r);
    float s, e1, u, e2;
    two_sum(pe, q, s, e1);
    two_sum(s, r, u, e2);
    return tf{p, u, __fadd_rn(__fmaf_rn(x.lo, y.lo, __fadd_rn(qe, re)), __fadd_rn(e1, e2))};
  }
  PP_D static T mul2(df x, df y, df u, df v) { return add(mul(x, y), mul(u, v)); }
  PP_D static T shfl_xor(T x, int o) {
    return tf{__shfl_xor_sync(0xffffffffu, x.a, o), __shfl_xor_sync(0xffffffffu, x.b, o),
              __shfl_xor_sync(0xffffffffu, x.c, o)};
  }
  PP_D static double to(T x) { return (double)x.a + ((double)x.b + (double)x.c); }
  PP_D static df toR(T x) {
    float s, e;
    two_sum(x.a, x.b, s, e);
    df r;
    fast_two_sum(s, __fadd_rn(e, x.c), r.hi, r.lo);
    return r;
  }
};
// a value of R from another lane
template <class R>
__device__ __forceinline__ R shfl_real(R x, int src) {
  R y;
  float *dst = (float *)&y;
  const float *p = (const float *)&x;
#pragma unroll
  for (int f = 0; f < (int)(sizeof(R) / sizeof(float)); ++f) dst[f] = __shfl_sync(0xffffffffu, p[f], src);
  return y;
}
// A complex sum over rows of products.  The double-float form keeps the products
// and the sums as three floats (2^-66 of the largest term, more than FP64): the sum
// does not depend on how the rows are dealt to lanes and CTAs, so a matrix gives
// the same result in a batch of any largest order.
template <class R>
struct __align__(16) RowSum {
  typename Sum<R>::T re, im;
  __device__ __forceinline__ void zero() { re = im = Sum<R>::zero(); }
  // += conj(w) v
  __device__ __forceinline__ void add_product(cx<R> w, cx<R> v) {
    re = Sum<R>::add(re, Sum<R>::mul2(w.re, v.re, w.im, v.im));
    im = Sum<R>::add(im, Sum<R>::mul2(w.re, v.im, RT<R>::neg(w.im), v.re));
  }
  __device__ __forceinline__ void add(const RowSum &o) {
    re = Sum<R>::add(re, o.re);
    im = Sum<R>::add(im, o.im);
  }
  // over lanes 0, 8, 16, 24 (the rows of a warp), in every one of them
  __device__ __forceinline__ void rows4() {
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) {
      re = Sum<R>::add(re, Sum<R>::shfl_xor(re, o));
      im = Sum<R>::add(im, Sum<R>::shfl_xor(im, o));
    }
  }
};
// -1/2 t s, s the sum of a warp's parts, in every lane: lanes 0-15 sum and form
// the real part, 16-31 the imaginary part; the product in FP64
template <class R>
__device__ __forceinline__ cx<R> minus_half_product(const RowSum<R> &part, z64 t) {
  typedef Sum<R> S;
  const bool im = (threadIdx.x & 31) >= 16;
  typename S::T v = S::add(im ? part.im : part.re, S::shfl_xor(im ? part.re : part.im, 16));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = S::add(v, S::shfl_xor(v, o));
  const double mine = S::to(v), other = __shfl_xor_sync(0xffffffffu, mine, 16);
  const double ts = im ? fma(t.im, other, t.re * mine) : fma(-t.im, other, t.re * mine);
  const R half = RT<R>::from(-0.5 * ts);
  return cx<R>{shfl_real(half, 0), shfl_real(half, 16)};
}

// 1/x, |x| in the middle of the exponent range: the hardware's estimate and one
// step of third order (Halley's iteration, r (1 + e + e^2) with e = 1 - x r): with
// |e| < 2^-19, r is off by less than 2^-57 relative before its one rounding, so at
// most 0.57 units in the last place (a correctly rounded quotient: 0.5).
// Three dependent FP64 operations where a division waits 560 cycles.
__device__ __forceinline__ double recip(double x) {
  if ((unsigned)((__double2hiint(x) >> 20 & 0x7ff) - 23) >= 2000u) return 1.0 / x;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

}  // namespace pp
