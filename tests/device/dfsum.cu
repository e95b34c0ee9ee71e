// The double-float multiply-adds, called from a test.
#include "../../parphom_gb300/csrc/pp_common.cuh"

#define EXPORT extern "C" __attribute__((visibility("default")))

// A thread per case: the sum of DF_BLOCK complex products a b (or conj(a) b) in one
// accumulator and as the mat-vec forms it.
__global__ void k_sums(int cases, int conj, const float4 *a, const float4 *b, float4 *one, float4 *two) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cases) return;
  auto at = [&](const float4 *v, int k) {
    const float4 x = v[c * DF_BLOCK + k];
    return zdf{df{x.x, x.y}, df{x.z, x.w}};
  };
  zdf s = cz<df>(), t = cz<df>();
  for (int k = 0; k < DF_BLOCK; ++k) {
    if (conj)
      cmacc(s, at(a, k), at(b, k));
    else
      cmac(s, at(a, k), at(b, k));
  }
  auto x = [&](int k) { return at(a, k); };
  auto y = [&](int k) { return at(b, k); };
  if (conj)
    df_block<true>(t, x, y);
  else
    df_block<false>(t, x, y);
  s = cfin(s);
  t = cfin(t);
  one[c] = make_float4(s.re.hi, s.re.lo, s.im.hi, s.im.lo);
  two[c] = make_float4(t.re.hi, t.re.lo, t.im.hi, t.im.lo);
}

EXPORT int sums(int cases, int conj, const float *a, const float *b, float *one, float *two) {
  k_sums<<<(cases + 63) / 64, 64>>>(cases, conj, (const float4 *)a, (const float4 *)b, (float4 *)one, (float4 *)two);
  return (int)cudaDeviceSynchronize();
}
