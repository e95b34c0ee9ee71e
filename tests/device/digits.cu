// The tensor-core products' digits and folds, called from a test.
#include "../../parphom_gb300/csrc/pp_digits.cuh"

#define EXPORT extern "C" __attribute__((visibility("default")))
using namespace pp;

// One warp per row of 64 values: its exponent and the 7 digits of each value.
__global__ void k_digits(const float *hi, const float *lo, int neg, int *E, float *dig) {
  const int row = blockIdx.x, lane = threadIdx.x;
  df x[2];
  for (int t = 0; t < 2; ++t) x[t] = df{hi[64 * row + 2 * lane + t], lo[64 * row + 2 * lane + t]};
  float amax = max_abs(fabsf(x[0].hi), x[1].hi);
  for (int o = 16; o > 0; o >>= 1) amax = max_abs(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const int e = grid_exp(amax);
  Fixed56 f[2];
  to_fixed<2>(x, e, neg != 0, f);
  const uint32_t w[7] = {digit2<0>(f[0], f[1]), digit2<1>(f[0], f[1]), digit2<2>(f[0], f[1]), digit2<3>(f[0], f[1]),
                         digit2<4>(f[0], f[1]), digit2<5>(f[0], f[1]), digit2<6>(f[0], f[1])};
  for (int s = 0; s < 7; ++s) {
    const __half2 h = *(const __half2 *)&w[s];
    dig[(7 * row + s) * 64 + 2 * lane] = __low2float(h);
    dig[(7 * row + s) * 64 + 2 * lane + 1] = __high2float(h);
  }
  if (lane == 0) E[row] = e;
}

// Both folds of 7 group sums, and the scale 2^(E - 16) of a product.
__global__ void k_fold(int n, const float *a, float *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float *g = a + 7 * i;
  df s, u;
  fold_group<6>(s, g[6]);
  fold_group<5>(s, g[5]);
  fold_group<4>(s, g[4]);
  fold_group<0>(s, g[0]);
  fold_group<1>(s, g[1]);
  fold_group<2>(s, g[2]);
  fold_group<3>(s, g[3]);
  s = fold_done(s);
  fold_up<6>(u, g[6]);
  fold_up<5>(u, g[5]);
  fold_up<4>(u, g[4]);
  fold_up<3>(u, g[3]);
  fold_up<2>(u, g[2]);
  fold_up<1>(u, g[1]);
  fold_up<0>(u, g[0]);
  out[4 * i] = s.hi;
  out[4 * i + 1] = s.lo;
  out[4 * i + 2] = u.hi;
  out[4 * i + 3] = u.lo;
}
__global__ void k_scale(int n, const int *e, float *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = pow2f(e[i]);
}

EXPORT int digits(int rows, const float *hi, const float *lo, int neg, int *E, float *dig) {
  k_digits<<<rows, 32>>>(hi, lo, neg, E, dig);
  return (int)cudaDeviceSynchronize();
}
EXPORT int fold(int n, const float *a, float *out) {
  k_fold<<<(n + 127) / 128, 128>>>(n, a, out);
  return (int)cudaDeviceSynchronize();
}
EXPORT int scale(int n, const int *e, float *out) {
  k_scale<<<(n + 127) / 128, 128>>>(n, e, out);
  return (int)cudaDeviceSynchronize();
}
