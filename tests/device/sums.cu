// The column step's sums, called from a test.
#include "../../parphom_gb300/csrc/pp_sums.cuh"

#define EXPORT extern "C" __attribute__((visibility("default")))
using namespace pp;

// One warp per case: lane l adds conj(w) v of entries l, l + 32, ...; the warp's
// -1/2 t (sum) and every lane's own sum (three floats each, real and imaginary).
__global__ void k_sums(int n, const float4 *w, const float4 *v, const double2 *t, float *own, float4 *out) {
  const int c = blockIdx.x, lane = threadIdx.x;
  RowSum<df> s;
  s.zero();
  for (int k = lane; k < n; k += 32) {
    const float4 a = w[c * n + k], b = v[c * n + k];
    s.add_product(zdf{df{a.x, a.y}, df{a.z, a.w}}, zdf{df{b.x, b.y}, df{b.z, b.w}});
  }
  const float f[6] = {s.re.a, s.re.b, s.re.c, s.im.a, s.im.b, s.im.c};
  for (int k = 0; k < 6; ++k) own[(c * 32 + lane) * 6 + k] = f[k];
  const zdf r = minus_half_product(s, z64{t[c].x, t[c].y});
  if (lane == 0) out[c] = make_float4(r.re.hi, r.re.lo, r.im.hi, r.im.lo);
}

__global__ void k_recip(int n, const double *x, double *r, double *q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = recip(x[i]);
  q[i] = 1.0 / x[i];
}

EXPORT int reciprocals(int n, const double *x, double *r, double *q) {
  k_recip<<<(n + 127) / 128, 128>>>(n, x, r, q);
  return (int)cudaDeviceSynchronize();
}
EXPORT int sums(int cases, int n, const float *w, const float *v, const double *t, float *own, float *out) {
  k_sums<<<cases, 32>>>(n, (const float4 *)w, (const float4 *)v, (const double2 *)t, own, (float4 *)out);
  return (int)cudaDeviceSynchronize();
}
