// Set-up of the default FP64 form: the per-point fixed-point weights K that
// heat_fp64_fx.cu reads (8 bytes per point), and the check that the form can
// represent the problem.

#include "heat_internal.h"

namespace heat {
namespace {

typedef unsigned long long u64;
typedef long long i64;

// K[c] = factor * kappa[c] rounded to 2^-63, from the error-free product
// p + q = factor * kappa (q = fma(factor, kappa, -p)), as two limbs
// k1 2^-32 + k0 2^-63 with |k0| <= 2^30: k1 in the high word, k0 (signed) in
// the low one.  Padding columns get 0.  bad[0] is set for negative or
// non-finite kappa and for factor * kappa >= 1/4.
// Bound: the FP64 pipe, 6 operations per point.
__global__ void k_kq_setup(u64 *__restrict__ K, int *__restrict__ bad,
                           const double *__restrict__ kap, int nx, int P, long rows,
                           double factor) {
  // One row per block iteration, its points across the threads.
  for (long r = blockIdx.x; r < rows; r += gridDim.x)
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
      const size_t c = (size_t)r * P + i;
      if (i >= nx) {
        K[c] = 0;
        continue;
      }
      const double kc = kap[c];
      const u64 bits = (u64)__double_as_longlong(kc);
      const double p = factor * kc, q = fma(factor, kc, -p);
      u64 v = 0;
      // finite and not negative (-0.0 is 0), p < 1/4
      if ((bits < 0x7ff0000000000000ull || bits << 1 == 0) && __double2hiint(p) < 0x3fd00000) {
        v = (u64)((i64)__double2ull_rn(p * 0x1p63) + __double2ll_rn(q * 0x1p63));
      } else {
        atomicOr(bad, 1);
      }
      const u64 k1 = (v + (1ull << 30)) >> 31;
      K[c] = (k1 << 32) | (unsigned)(v - (k1 << 31));
    }
}

// bad[0] is set where a centre weight 1 - sum_f w_f is below 2^-40, or the high limbs of
// the six weights sum to more than 1 (low limbs below zero; only for centre weights below
// 7 x 2^-32).  With neither, no sum of the fixed-point form leaves 64 bits: a result is a
// mean of values, and the sum of d0 w1 stays below 2^32 (2^32 - 1) + 2^31.
__global__ void k_kq_check(const u64 *__restrict__ K, int *__restrict__ bad, int nx, int ny, int nz,
                           int P, size_t S) {
  bool ok = true;
  const long rows = (long)(ny - 2) * (nz - 2);
  for (long r = blockIdx.x; r < rows; r += gridDim.x) {
    const size_t row = (size_t)(1 + r / (ny - 2)) * S + (size_t)(1 + r % (ny - 2)) * P;
    for (int i = 1 + threadIdx.x; i < nx - 1; i += blockDim.x) {
      const u64 *k = K + row + i;
      u64 s1 = 6 * (*k >> 32);             // units of 2^-32
      i64 s0 = 6ll * (int)(unsigned)*k;    // of 2^-63
      for (const u64 v : {k[1], k[-1], k[P], k[-(ptrdiff_t)P], k[S], k[-(ptrdiff_t)S]}) {
        s1 += v >> 32;
        s0 += (int)(unsigned)v;
      }
      ok &= s1 <= 1ull << 32 && (s1 << 31) + (u64)s0 <= (1ull << 63) - (1ull << 23);
    }
  }
  if (!ok) atomicOr(bad, 1);
}

}  // namespace

cudaError_t launch_kq_setup(unsigned long long *K, int *bad, const double *kappa,
                            const heat_geom &g, double factor, cudaStream_t st) {
  k_kq_setup<<<152 * 8, 256, 0, st>>>(K, bad, kappa, g.nx, g.pitch, (long)g.ny * g.nz, factor);
  k_kq_check<<<152 * 8, 256, 0, st>>>(K, bad, g.nx, g.ny, g.nz, g.pitch, g.plane);
  return cudaGetLastError();
}

}  // namespace heat
