// Density of states from the frequencies of a q-grid: linear triangulation
// and Gaussian / Lorentzian smearing, restated from the reference's
// BZ-integration routines (Utilities/pyphutil/fortran_routines/
// bz_integration.f90:12-48, 50-65, 68-133, 154-199).
//
// Triangulation: for each energy E, triangle and band, the four values
// (E with weight 0 and the band's frequencies at the three vertices with
// their weights f) are sorted by value with the same exchange sort; the
// position E takes decides the closed-form contribution (dos, nd) of that
// triangle, with the same case order (position 4, 3, 2, 1; a later case
// overrides an earlier one when values tie).  k_dos_tri takes 32 triangles of
// a band per warp.  FP64 throughout.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>

#include "../../include/parphom_gpu.h"
#include "pp_internal.cuh"

namespace {

constexpr double PI_REF = (double)3.141592653589793f;  // bz_integration.f90:185, 195

__device__ void integrate_triangle(const double a[4][2], double Ef, double &dos, double &nd) {
  dos = 0.0;
  nd = 0.0;
  if (a[3][0] == Ef) {
    dos = 0.0;
    nd = a[0][1] + a[1][1] + a[2][1];
  }
  if (a[2][0] == Ef) {
    const double e0 = a[0][0], f0 = a[0][1], e1 = a[1][0], f1 = a[1][1], e2 = a[3][0], f2 = a[3][1];
    const double del02 = (e2 - Ef) / (e2 - e0), del12 = (e2 - Ef) / (e2 - e1);
    const double ddel02 = 1 / (e0 - e2), ddel12 = 1 / (e1 - e2);
    nd = (1 - del12 * (del02 * del02)) * f0 + (1 - del02 * (del12 * del12)) * f1 +
         (1 - 3 * del12 * del02 + del12 * (del02 * del02) + del02 * (del12 * del12)) * f2;
    dos = (-2 * del02 * ddel02 * del12 - ddel12 * (del02 * del02)) * f0 +
          (-ddel02 * (del12 * del12) - 2 * del02 * del12 * ddel12) * f1 +
          (-3 * del12 * ddel02 - 3 * del02 * ddel12 + 2 * del02 * del12 * ddel02 + ddel12 * (del02 * del02) +
           2 * del02 * del12 * ddel12 + ddel02 * (del12 * del12)) *
              f2;
  }
  if (a[1][0] == Ef) {
    const double e0 = a[0][0], f0 = a[0][1], e1 = a[2][0], f1 = a[2][1], e2 = a[3][0], f2 = a[3][1];
    const double del10 = (Ef - e0) / (e1 - e0), del20 = (Ef - e0) / (e2 - e0);
    const double ddel10 = 1 / (e1 - e0), ddel20 = 1 / (e2 - e0);
    double n = (3 - del10 - del20) * f0 + del10 * f1 + del20 * f2;
    dos = ddel10 * del20 * n + del10 * ddel20 * n + del10 * del20 * ((-ddel10 - ddel20) * f0 + ddel10 * f1 + ddel20 * f2);
    nd = n * del10 * del20;
  }
  if (a[0][0] == Ef) {
    dos = 0.0;
    nd = 0.0;
  }
}

// One triangle and band by the sort itself: energies that tie with a vertex,
// and values that do not compare.
__device__ __noinline__ void triangle_by_sort(const double *freq, int64_t ldf, const double *func, int64_t ldfunc,
                                              const int64_t *tri, int64_t k, double Ef, double &d, double &n) {
  double a[4][2];
  a[0][0] = Ef;
  a[0][1] = 0.0;
  for (int v = 0; v < 3; ++v) {
    const int64_t q = tri[v];
    a[v + 1][0] = freq[q * ldf + k];
    a[v + 1][1] = func ? func[q * ldfunc + k] : 1.0;
  }
  for (int p = 0; p < 4; ++p)  // exchange sort of bz_integration.f90:50-65
    for (int r = p + 1; r < 4; ++r)
      if (a[p][0] > a[r][0]) {
        const double t0 = a[p][0], t1 = a[p][1];
        a[p][0] = a[r][0];
        a[p][1] = a[r][1];
        a[r][0] = t0;
        a[r][1] = t1;
      }
  integrate_triangle(a, Ef, d, n);
}

// Sums over triangles and bands.  A warp takes 32 triangles of one band, a
// lane one of them, its vertices sorted and the three reciprocals taken once.
// Most energies lie above all 32 triangles (they add the warp's weights to nd)
// or below (nothing): lanes then stand for energies, 32 at a time.  For the few
// in between, lanes stand for triangles.  Each warp adds to sums of its own in
// shared memory (DT_E energies); a block's go to part ([dos, nd][energy][block]) at
// the end, which k_dos_sum adds up, or without part are added to dos / nd one after
// the other (32 x 32 grid, 444 bands, rms: dos off by 2.4e-16 and nd by 2.3e-16 that
// way, by 1.0e-16 both with part).
//
// Bound by the FP64 pipe (16 cycles per instruction of a warp): two comparisons
// per 32 energies and about 40 instructions per energy in between, no division.
// A thread per (energy, band) that sorted and evaluated every triangle took
// 33.6 ms for 1024 q-points, 444 bands and 1000 energies; this takes 1.8 ms.
constexpr int DT_W = 16;    // warps per block
constexpr int DT_E = 512;   // energies per block
constexpr int DT_SMEM = (2 * DT_W + 1) * DT_E * 8;
__global__ void __launch_bounds__(32 * DT_W, 1) k_dos_tri(const double *freq, int64_t ldf, const double *func,
                                                          int64_t ldfunc, int64_t nbands, const int64_t *tri,
                                                          int64_t ntri, const double *E, int64_t ne, double *dos,
                                                          double *nd, double *part) {
  extern __shared__ double sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *sE = sm, *sd = sm + DT_E + 2 * DT_E * warp, *sn = sd + DT_E;
  const int64_t i0 = (int64_t)blockIdx.y * DT_E;
  const int nE = (int)(ne - i0 < DT_E ? ne - i0 : DT_E), nS = (nE + 31) / 32;
  for (int i = threadIdx.x; i < DT_E; i += 32 * DT_W) sE[i] = i < nE ? E[i0 + i] : 0.0;
  for (int i = lane; i < 2 * DT_E; i += 32) sd[i] = 0.0;
  __syncthreads();
  const int64_t items = (ntri + 31) / 32 * nbands;
  for (int64_t it = (int64_t)blockIdx.x * DT_W + warp; it < items; it += (int64_t)gridDim.x * DT_W) {
    const int64_t k = it % nbands, j = it / nbands * 32 + lane;
    const bool have = j < ntri;
    double e0 = INFINITY, e1 = INFINITY, e2 = INFINITY, f0 = 0.0, f1 = 0.0, f2 = 0.0;
    bool odd = false;  // values that do not compare
    if (have) {
      const int64_t q0 = tri[3 * j], q1 = tri[3 * j + 1], q2 = tri[3 * j + 2];
      e0 = freq[q0 * ldf + k];
      e1 = freq[q1 * ldf + k];
      e2 = freq[q2 * ldf + k];
      f0 = func ? func[q0 * ldfunc + k] : 1.0;
      f1 = func ? func[q1 * ldfunc + k] : 1.0;
      f2 = func ? func[q2 * ldfunc + k] : 1.0;
      odd = isnan(e0) || isnan(e1) || isnan(e2);
      auto order = [](double &a, double &fa, double &b, double &fb) {
        const bool g = a > b;
        const double t = a, tf = fa;
        a = g ? b : a;
        fa = g ? fb : fa;
        b = g ? t : b;
        fb = g ? tf : fb;
      };
      order(e0, f0, e1, f1);
      order(e1, f1, e2, f2);
      order(e0, f0, e1, f1);
    }
    const double r10 = 1.0 / (e1 - e0), r20 = 1.0 / (e2 - e0), r21 = 1.0 / (e2 - e1);
    // (values so close that a reciprocal overflows: by quotients as well)
    auto inf = [](double x) { return (__double2hiint(x) & 0x7fffffff) == 0x7ff00000; };
    odd = odd || (inf(r10) && e1 > e0) || (inf(r21) && e2 > e1);
    const double fs = f0 + f1 + f2;
    double lo = odd ? -INFINITY : e0, hi = odd ? INFINITY : have ? e2 : -INFINITY, all = fs;
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    for (int st = 0; st < nS; ++st) {
      const int i = 32 * st + lane;
      const double mine = sE[i];
      const bool above = mine > hi, inside = i < nE && !above && !(mine <= lo);
      if (above) sn[i] += all;
      for (unsigned todo = __ballot_sync(0xffffffffu, inside); todo; todo &= todo - 1) {
        const int l = __ffs((int)todo) - 1;
        const double Ef = __shfl_sync(0xffffffffu, mine, l);
        double d = 0.0, n = 0.0;
        if (have && !(Ef <= e0 && !odd)) {
          if (Ef > e2 && !odd) {
            n = fs;
          } else if (Ef > e0 && Ef < e1 && !odd) {
            const double x = Ef - e0, del10 = x * r10, del20 = x * r20;
            const double m = (3 - del10 - del20) * f0 + del10 * f1 + del20 * f2;
            d = r10 * del20 * m + del10 * r20 * m + del10 * del20 * ((-r10 - r20) * f0 + r10 * f1 + r20 * f2);
            n = m * del10 * del20;
          } else if (Ef > e1 && Ef < e2 && !odd) {
            const double x = e2 - Ef, del02 = x * r20, del12 = x * r21, ddel02 = -r20, ddel12 = -r21;
            n = (1 - del12 * (del02 * del02)) * f0 + (1 - del02 * (del12 * del12)) * f1 +
                (1 - 3 * del12 * del02 + del12 * (del02 * del02) + del02 * (del12 * del12)) * f2;
            d = (-2 * del02 * ddel02 * del12 - ddel12 * (del02 * del02)) * f0 +
                (-ddel02 * (del12 * del12) - 2 * del02 * del12 * ddel12) * f1 +
                (-3 * del12 * ddel02 - 3 * del02 * ddel12 + 2 * del02 * del12 * ddel02 + ddel12 * (del02 * del02) +
                 2 * del02 * del12 * ddel12 + ddel02 * (del12 * del12)) *
                    f2;
          } else {
            triangle_by_sort(freq, ldf, func, ldfunc, tri + 3 * j, k, Ef, d, n);
          }
        }
        for (int o = 16; o > 0; o >>= 1) {
          d += __shfl_xor_sync(0xffffffffu, d, o);
          n += __shfl_xor_sync(0xffffffffu, n, o);
        }
        if (lane == l) {
          sd[i] += d;
          sn[i] += n;
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nE; i += 32 * DT_W) {
    double d = 0.0, n = 0.0;
    for (int w = 0; w < DT_W; ++w) {
      d += sm[DT_E + 2 * DT_E * w + i];
      n += sm[DT_E + 2 * DT_E * w + DT_E + i];
    }
    if (part) {
      part[(i0 + i) * gridDim.x + blockIdx.x] = d;
      part[(ne + i0 + i) * gridDim.x + blockIdx.x] = n;
    } else {
      atomicAdd(&dos[i0 + i], d);
      atomicAdd(&nd[i0 + i], n);
    }
  }
}
// one block per SM and slice of energies, fewer for fewer groups of triangles
unsigned dos_tri_blocks(int64_t ntri, int64_t nbands, int64_t ne) {
  const int64_t items = (ntri + 31) / 32 * nbands, slices = (ne + DT_E - 1) / DT_E;
  const int64_t per = std::max<int64_t>(1, pp::device_sms() / std::min<int64_t>(slices, pp::device_sms()));
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((items + DT_W - 1) / DT_W, per));
}
// The blocks' parts of dos and nd added up: a warp per sum, its lanes' parts by a
// tree, so that few additions round at the size of the total (carrying their
// rounding errors along as well: 0.88e-16 instead of 0.95e-16, 2 us more a call).
__global__ void __launch_bounds__(128) k_dos_sum(const double *part, int nblk, int64_t ne, double *dos, double *nd) {
  const int64_t i = (int64_t)blockIdx.x * 4 + threadIdx.x / 32;
  const int lane = threadIdx.x & 31;
  if (i >= 2 * ne) return;
  double s = 0.0;
  for (int k = lane; k < nblk; k += 32) s += part[i * nblk + k];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) (i < ne ? dos : nd)[i < ne ? i : i - ne] = s;
}

// dos and nd with the blocks' parts in `part` (2 ne dos_tri_blocks doubles), or
// without.
cudaError_t dos_tri(const double *freq, int64_t ldf, const double *func, int64_t ldfunc, int64_t nbands,
                    const int64_t *tri, int64_t ntri, const double *E, int64_t ne, double *dos, double *nd,
                    double *part, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(k_dos_tri, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_SMEM);
  if (e == cudaSuccess && !part) e = cudaMemsetAsync(dos, 0, sizeof(double) * ne, s);
  if (e == cudaSuccess && !part) e = cudaMemsetAsync(nd, 0, sizeof(double) * ne, s);
  if (e != cudaSuccess) return e;
  const unsigned nblk = dos_tri_blocks(ntri, nbands, ne);
  k_dos_tri<<<dim3(nblk, (unsigned)((ne + DT_E - 1) / DT_E)), 32 * DT_W, DT_SMEM, s>>>(
      freq, ldf, func, ldfunc, nbands, tri, ntri, E, ne, dos, nd, part);
  if (part) k_dos_sum<<<(unsigned)((2 * ne + 3) / 4), 128, 0, s>>>(part, (int)nblk, ne, dos, nd);
  pp::count_launch(part ? 2 : 1);
  return cudaGetLastError();
}

// Room for the parts of the device-resident form, which allocates nothing: fixed
// arrays of the library, one for each of up to DS_SLOTS streams with calls in flight
// on a device.  A call takes the array that its stream used last, or the one unused
// for longest, whose last call it waits for on the device; inside a stream capture (a
// graph may run at any time) and past DS_CAP it goes without.
constexpr int DS_SLOTS = 2;
constexpr int64_t DS_CAP = 2 * 160 * DT_E;  // doubles: 160 SMs with DT_E energies each
__device__ double dos_parts[DS_SLOTS][DS_CAP];
struct DosSlots {
  double *base = nullptr;
  cudaStream_t stream[DS_SLOTS] = {};
  cudaEvent_t done[DS_SLOTS] = {};
  uint64_t used[DS_SLOTS] = {}, uses = 0;  // 0: never
};
std::mutex ds_mu;
DosSlots ds_slots[pp::PP_MAX_DEVICES];

// launch(part) with a slot's array or with nullptr
template <class F>
cudaError_t with_parts(int64_t need, cudaStream_t s, F launch) {
  const int dev = pp::device_index();
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {  // (the legacy stream while another is captured)
    cudaGetLastError();
    cs = cudaStreamCaptureStatusActive;
  }
  if (dev < 0 || need > DS_CAP || cs != cudaStreamCaptureStatusNone) return launch(nullptr);
  std::lock_guard<std::mutex> g(ds_mu);
  DosSlots &d = ds_slots[dev];
  if (!d.base) {
    // (another thread may be capturing: neither call touches its stream)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, dos_parts);
    for (int k = 0; k < DS_SLOTS && e == cudaSuccess; ++k)
      if (!d.done[k]) e = cudaEventCreateWithFlags(&d.done[k], cudaEventDisableTiming);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return e;
    d.base = (double *)p;
  }
  int k = 0;
  for (int t = 1; t < DS_SLOTS; ++t)
    if (d.used[t] < d.used[k]) k = t;
  for (int t = 0; t < DS_SLOTS; ++t)
    if (d.used[t] && d.stream[t] == s) k = t;
  cudaError_t e = d.used[k] ? cudaStreamWaitEvent(s, d.done[k], 0) : cudaSuccess;
  if (e != cudaSuccess) return e;
  e = launch(d.base + k * DS_CAP);
  d.used[k] = ++d.uses;
  d.stream[k] = s;
  const cudaError_t r = cudaEventRecord(d.done[k], s);
  return e != cudaSuccess ? e : r;
}

__global__ void k_dos_smear(int method, const double *freq, int64_t ldf, int64_t nq, int64_t nbands,
                            const double *weights, double width, const double *E, int64_t ne, double *pdos) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // band
  const int64_t i = blockIdx.y;
  if (k >= nbands || i >= ne) return;
  const double e = E[i];
  double s = 0.0;
  for (int64_t q = 0; q < nq; ++q) {
    const double e0 = freq[q * ldf + k];
    double d;
    if (method == 1) {
      const double x = (e - e0) / width;
      d = exp(-(x * x) / 2) / (sqrt(2 * PI_REF) * width);
    } else {
      const double h = width / 2;
      d = (h / ((e - e0) * (e - e0) + h * h)) * (1 / PI_REF);
    }
    s += d * weights[q];
  }
  pdos[i * nbands + k] = s;
}

__global__ void k_sum_rows(const double *p, int64_t ne, int64_t nb, double scale, double *out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ne) return;
  double s = 0.0;
  for (int64_t k = 0; k < nb; ++k) s += p[i * nb + k];
  out[i] = s * scale;
}

int cerr(cudaError_t e) { return e == cudaSuccess ? PP_OK : (e == cudaErrorMemoryAllocation ? PP_ERR_NOMEM : PP_ERR_CUDA); }

// ---- device-resident forms: every array in device memory, no scratch.
// One thread per band, one block row per energy; the block's bands are
// summed in shared memory and added to the energy's total (zeroed first).
constexpr int DV_NT = 128;

__device__ __forceinline__ double block_sum128(double v, double *sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < DV_NT / 32; ++k) r += sh[k];
  return r;  // valid in thread 0
}

__global__ void __launch_bounds__(DV_NT) k_dos_smear_dev(int method, const double *freq, int64_t ldf, int64_t nq,
                                                         int64_t nbands, const double *weights, double width,
                                                         const double *E, int64_t ne, double scale, double *dos) {
  __shared__ double sh[DV_NT / 32];
  const int64_t k = (int64_t)blockIdx.x * DV_NT + threadIdx.x;
  const int64_t i = blockIdx.y;
  if (i >= ne) return;
  const double e = E[i];
  double s = 0.0;
  if (k < nbands) {
    for (int64_t q = 0; q < nq; ++q) {
      const double e0 = freq[q * ldf + k];
      double d;
      if (method == 1) {
        const double x = (e - e0) / width;
        d = exp(-(x * x) / 2) / (sqrt(2 * PI_REF) * width);
      } else {
        const double h = width / 2;
        d = (h / ((e - e0) * (e - e0) + h * h)) * (1 / PI_REF);
      }
      s += d * weights[q];
    }
  }
  s = block_sum128(s, sh);
  if (threadIdx.x == 0) atomicAdd(&dos[i], s * scale);
}

// func[q ldfunc + j] = v_a v_b of mode j at q-point q (a = b = -1: |v|^2),
// from the velocity output vel[q velstride + 3 j + d].
__global__ void k_vel_weights(const double *vel, int64_t velstride, int64_t nq, int64_t nbands, int a, int b,
                              double *func, int64_t ldfunc) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t q = blockIdx.y;
  if (j >= nbands || q >= nq) return;
  const double *v = vel + q * velstride + 3 * j;
  func[q * ldfunc + j] = (a < 0) ? v[0] * v[0] + v[1] * v[1] + v[2] * v[2] : v[a] * v[b];
}

}  // namespace

extern "C" PP_API int pp_dos_triangulation(const double *freq, int64_t ldf, int64_t nk, int64_t nbands,
                                           const double *func, const int64_t *tri, int64_t ntri, const double *energy,
                                           int64_t ne, double *dos, double *nd) {
  if (!freq) return -1;
  if (ldf < nbands) return -2;
  if (nk < 1) return -3;
  if (nbands < 1) return -4;
  if (!tri && ntri > 0) return -6;
  if (ntri < 0) return -7;
  if (!energy && ne > 0) return -8;
  if (ne < 0) return -9;
  if (!dos) return -10;
  if (!nd) return -11;
  for (int64_t j = 0; j < 3 * ntri; ++j)
    if (tri[j] < 0 || tri[j] >= nk) return -6;
  if (ne == 0) return PP_OK;
  double *dfreq = nullptr, *dfunc = nullptr, *dE = nullptr, *part = nullptr, *od = nullptr, *on = nullptr;
  int64_t *dtri = nullptr;
  cudaError_t e = cudaSuccess;
  auto al = [&](void **p, size_t b) {
    if (e == cudaSuccess) e = cudaMalloc(p, b > 0 ? b : 8);
  };
  al((void **)&dfreq, sizeof(double) * nk * ldf);
  if (func) al((void **)&dfunc, sizeof(double) * nk * ldf);
  al((void **)&dtri, sizeof(int64_t) * 3 * ntri);
  al((void **)&dE, sizeof(double) * ne);
  al((void **)&part, sizeof(double) * 2 * ne * dos_tri_blocks(ntri, nbands, ne));
  al((void **)&od, sizeof(double) * ne);
  al((void **)&on, sizeof(double) * ne);
  if (e == cudaSuccess) e = cudaMemcpy(dfreq, freq, sizeof(double) * nk * ldf, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && func) e = cudaMemcpy(dfunc, func, sizeof(double) * nk * ldf, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && ntri) e = cudaMemcpy(dtri, tri, sizeof(int64_t) * 3 * ntri, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dE, energy, sizeof(double) * ne, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = dos_tri(dfreq, ldf, dfunc, ldf, nbands, dtri, ntri, dE, ne, od, on, part, 0);
  if (e == cudaSuccess) e = cudaMemcpy(dos, od, sizeof(double) * ne, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(nd, on, sizeof(double) * ne, cudaMemcpyDeviceToHost);
  for (void *p : {(void *)dfreq, (void *)dfunc, (void *)dtri, (void *)dE, (void *)part, (void *)od, (void *)on})
    if (p) cudaFree(p);
  return cerr(e);
}

extern "C" PP_API int pp_dos_smearing(int32_t method, const double *freq, int64_t ldf, int64_t nq, int64_t nbands,
                                      const double *weights, double width, const double *energy, int64_t ne,
                                      int64_t natom, double *dos) {
  if (method != 1 && method != 2) return -1;
  if (!freq) return -2;
  if (ldf < nbands) return -3;
  if (nq < 1) return -4;
  if (nbands < 1) return -5;
  if (!weights) return -6;
  if (!(width > 0.0)) return -7;
  if (!energy && ne > 0) return -8;
  if (ne < 0) return -9;
  if (natom < 1) return -10;
  if (!dos) return -11;
  if (ne == 0) return PP_OK;
  double *dfreq = nullptr, *dw = nullptr, *dE = nullptr, *pd = nullptr, *od = nullptr;
  cudaError_t e = cudaSuccess;
  auto al = [&](void **p, size_t b) {
    if (e == cudaSuccess) e = cudaMalloc(p, b);
  };
  al((void **)&dfreq, sizeof(double) * nq * ldf);
  al((void **)&dw, sizeof(double) * nq);
  al((void **)&dE, sizeof(double) * ne);
  al((void **)&pd, sizeof(double) * ne * nbands);
  al((void **)&od, sizeof(double) * ne);
  if (e == cudaSuccess) e = cudaMemcpy(dfreq, freq, sizeof(double) * nq * ldf, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dw, weights, sizeof(double) * nq, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dE, energy, sizeof(double) * ne, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_dos_smear<<<dim3((unsigned)((nbands + 127) / 128), (unsigned)ne), 128>>>(method, dfreq, ldf, nq, nbands, dw,
                                                                              width, dE, ne, pd);
    k_sum_rows<<<(unsigned)((ne + 127) / 128), 128>>>(pd, ne, nbands, 1.0 / (double)natom, od);
    pp::count_launch(2);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(dos, od, sizeof(double) * ne, cudaMemcpyDeviceToHost);
  for (void *p : {(void *)dfreq, (void *)dw, (void *)dE, (void *)pd, (void *)od})
    if (p) cudaFree(p);
  return cerr(e);
}

extern "C" PP_API int pp_dos_triangulation_device(const double *freq_dev, int64_t ldf, int64_t nk, int64_t nbands,
                                                  const double *func_dev, int64_t ldfunc, const int64_t *tri_dev,
                                                  int64_t ntri, const double *energy_dev, int64_t ne, double *dos_dev,
                                                  double *nd_dev, void *stream) {
  if (!freq_dev) return -1;
  if (ldf < nbands) return -2;
  if (nk < 1) return -3;
  if (nbands < 1) return -4;
  if (func_dev && ldfunc < nbands) return -6;
  if (!tri_dev && ntri > 0) return -7;
  if (ntri < 0) return -8;
  if (!energy_dev && ne > 0) return -9;
  if (ne < 0) return -10;
  if (!dos_dev) return -11;
  if (!nd_dev) return -12;
  if (ne == 0) return PP_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const cudaError_t e = with_parts(2 * ne * dos_tri_blocks(ntri, nbands, ne), s, [&](double *part) {
    return dos_tri(freq_dev, ldf, func_dev, ldfunc, nbands, tri_dev, ntri, energy_dev, ne, dos_dev, nd_dev, part, s);
  });
  return cerr(e);
}

extern "C" PP_API int pp_dos_smearing_device(int32_t method, const double *freq_dev, int64_t ldf, int64_t nq,
                                             int64_t nbands, const double *weights_dev, double width,
                                             const double *energy_dev, int64_t ne, int64_t natom, double *dos_dev,
                                             void *stream) {
  if (method != 1 && method != 2) return -1;
  if (!freq_dev) return -2;
  if (ldf < nbands) return -3;
  if (nq < 1) return -4;
  if (nbands < 1) return -5;
  if (!weights_dev) return -6;
  if (!(width > 0.0)) return -7;
  if (!energy_dev && ne > 0) return -8;
  if (ne < 0) return -9;
  if (natom < 1) return -10;
  if (!dos_dev) return -11;
  if (ne == 0) return PP_OK;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(dos_dev, 0, sizeof(double) * ne, s);
  if (e == cudaSuccess) {
    k_dos_smear_dev<<<dim3((unsigned)((nbands + DV_NT - 1) / DV_NT), (unsigned)ne), DV_NT, 0, s>>>(
        method, freq_dev, ldf, nq, nbands, weights_dev, width, energy_dev, ne, 1.0 / (double)natom, dos_dev);
    pp::count_launch(1);
    e = cudaGetLastError();
  }
  return cerr(e);
}

extern "C" PP_API int pp_velocity_weights_device(const double *vel_dev, int64_t velstride, int64_t nq, int64_t nbands,
                                                 int32_t a, int32_t b, double *func_dev, int64_t ldfunc,
                                                 void *stream) {
  if (!vel_dev) return -1;
  if (velstride < 3 * nbands) return -2;
  if (nq < 0) return -3;
  if (nbands < 1) return -4;
  if (!((a == -1 && b == -1) || (a >= 0 && a < 3 && b >= 0 && b < 3))) return -5;
  if (!func_dev) return -7;
  if (ldfunc < nbands) return -8;
  if (nq == 0) return PP_OK;
  cudaStream_t s = (cudaStream_t)stream;
  k_vel_weights<<<dim3((unsigned)((nbands + 127) / 128), (unsigned)nq), 128, 0, s>>>(vel_dev, velstride, nq, nbands,
                                                                                     a, b, func_dev, ldfunc);
  pp::count_launch(1);
  return cerr(cudaGetLastError());
}
