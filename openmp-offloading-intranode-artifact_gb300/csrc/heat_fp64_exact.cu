// Bit-exact FP64 kernels: the reference's operation order with every
// operation rounded separately (no fused multiply-add).  This translation unit
// is compiled with --fmad=false, and the arithmetic is written with the
// explicit round-to-nearest intrinsics (__dadd_rn, __dsub_rn, __dmul_rn),
// which the compiler never contracts, so the result does not depend on the
// contraction flag either way.
//
// Reference expression (OpenMP_Single_Source/heat3D_variable_coeff.c:174-181,
// 1-cuda.cu:103-111):
//   u_new = (u + rhs) + factor * S,
//   S = ((((A - B) + C) - D) + E) - F,
//   A = (kE+kC)(uE-uC)  B = (kC+kW)(uC-uW)  C = (kN+kC)(uN-uC)
//   D = (kC+kS)(uC-uS)  E = (kU+kC)(uU-uC)  F = (kC+kD)(uC-uD)
// A face flux is the same rounded value seen from both cells that share the
// face (IEEE addition is commutative), so the z-march below carries E of
// plane k as F of plane k+1 and stays bit-identical.

#include "heat_internal.h"
#include "heat_walk.cuh"

namespace heat {
namespace {

typedef unsigned long long u64;
using walk::combine;
using walk::flux;

// One thread per point, the reference CUDA kernel's shape (block 8x8x8,
// 1-cuda.cu:85-131), arbitrary row pitch.
template <bool RHS>
__global__ void k_naive(double *__restrict__ un, const double *__restrict__ u,
                        const double *__restrict__ rhs, const double *__restrict__ kap,
                        int nx, int ny, int nz, int P, size_t S, double factor) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  int k = blockIdx.z * blockDim.z + threadIdx.z;
  if (k < 1 || k >= nz - 1 || j < 1 || j >= ny - 1 || i < 1 || i >= nx - 1) return;
  size_t c = (size_t)k * S + (size_t)j * P + i;
  double uc = u[c], kc = kap[c];
  double A = flux(__dadd_rn(kap[c + 1], kc), u[c + 1], uc);
  double B = flux(__dadd_rn(kc, kap[c - 1]), uc, u[c - 1]);
  double C = flux(__dadd_rn(kap[c + P], kc), u[c + P], uc);
  double D = flux(__dadd_rn(kc, kap[c - P]), uc, u[c - P]);
  double E = flux(__dadd_rn(kap[c + S], kc), u[c + S], uc);
  double F = flux(__dadd_rn(kc, kap[c - S]), uc, u[c - S]);
  un[c] = combine(RHS ? __dadd_rn(uc, rhs[c]) : uc, factor, A, B, C, D, E, F);
}

__device__ __forceinline__ u64 shr(u64 a, unsigned n) {  // 0 for n >= 64
  u64 r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(n));
  return r;
}
// A conductivity as an integer with its leading bit at 62, so that a sum of two
// fits, and its exponent field.  Zeros and subnormals (a plain significand beside
// the field 0) need no care in a sum that is in range; negative values are odd.
struct Int {
  u64 m;
  unsigned e;
};
__device__ __forceinline__ Int integer(double v, bool &odd) {
  const unsigned hi = (unsigned)__double2hiint(v);
  odd |= (int)hi < 0;
  const unsigned h = (hi & 0xfffffu) | min(hi & 0x7ff00000u, 0x100000u);
  return {(((u64)h << 32) | (unsigned)__double2loint(v)) << 10, hi >> 20};
}

// A sum of two conductivities in [2^-200, 2^200): exponent field (in place) and
// significand, its leading bit at 63.
struct Weight {
  unsigned h, l, t;
};
__device__ __forceinline__ Weight weight(double k, bool &odd) {
  const unsigned hi = (unsigned)__double2hiint(k), lo = (unsigned)__double2loint(k);
  odd |= hi - (823u << 20) >= (400u << 20);
  return {__funnelshift_l(lo, hi, 11) | 0x80000000u, lo << 11, hi & 0x7ff00000u};
}
// fl(a + b).  Where an operand is shifted by more than its 10 zero bits the sum
// lacks less than a unit, which matters to the rounding of a tie only: odd, as a
// sum that rounds up to a power of two.
__device__ __forceinline__ Weight sum(const Int &a, const Int &b, bool &odd) {
  const unsigned e = max(a.e, b.e), da = e - a.e, db = e - b.e;
  const u64 s = shr(a.m, da) + shr(b.m, db);
  const unsigned n = (unsigned)(s >> 63) ^ 1, t = (e + 1 - n) << 20;
  const u64 x = s << n, y = x + 0x3ff + (x >> 11 & 1);
  odd |= y < x || (da + db > 10 && (x & 0x7ff) == 0x400) || t - (823u << 20) >= (400u << 20);
  return {(unsigned)(y >> 32), (unsigned)y & ~0x7ffu, t};
}
// fl(k d), for d zero or of a size in [2^-723, 2^677).  The 106-bit product of the
// significands keeps its first 53 bits; the next 32, and an or of the rest below
// them, round to nearest even through a carry that may run on into the exponent
// field.
__device__ __forceinline__ double product(const Weight &k, double d, bool &odd) {
  const unsigned hi = (unsigned)__double2hiint(d), a0 = (unsigned)__double2loint(d);
  const unsigned t = hi & 0x7ff00000u, a1 = (hi & 0xfffffu) | 0x100000u;
  const u64 p00 = (u64)a0 * k.l, p01 = (u64)a0 * k.h + (p00 >> 32);
  const u64 p10 = (u64)a1 * k.l + (unsigned)p01;
  const u64 p11 = (u64)a1 * k.h + (p01 >> 32) + (p10 >> 32);
  const unsigned h1 = (unsigned)(p11 >> 32), h0 = (unsigned)p11, l1 = (unsigned)p10;
  const unsigned top = h1 & 0x100000u, n = (top >> 20) ^ 1;
  const unsigned m1 = __funnelshift_l(h0, h1, n), m0 = __funnelshift_l(l1, h0, n);
  const unsigned x = __funnelshift_l((unsigned)p00, l1, n) | ((unsigned)p00 >> 11);
  const u64 carry = ((u64)x + 0x7fffffffu + (m0 & 1)) >> 32;
  u64 r = (((u64)m1 << 32) | m0) + carry + ((u64)(t + k.t + top - (1024u << 20)) << 32);
  if (t == 0) r = 0;
  odd |= t - (300u << 20) > (1400u << 20) && ((hi << 1) | a0) != 0;
  return __hiloint2double((int)((unsigned)(r >> 32) | (hi & 0x80000000u)), (int)(unsigned)r);
}

// z-marching kernel.  A thread walks a chunk of planes; it owns one column i of RY
// adjacent rows, and the lower flux and the z-neighbours of each row stay in
// registers.  Two face fluxes are shared instead of recomputed (a face flux is the
// same rounded value seen from both cells that share the face):
//   - x: B at column i is A of column i-1 (same operands, same order), taken
//     from the neighbouring lane.
//   - y: C of row j is D of row j+1, so a thread computes RY+1 y-fluxes for
//     its RY outputs instead of 2 RY.  Row t of a thread (t = 0 .. RY+1) is
//     grid row j0-1+t; rows past the grid are clamped to the last row so every
//     load stays in bounds, and only interior rows store (an interior row reads
//     rows j-1, j, j+1 only, none of them clamped).
// Columns 0 .. nx-2 of each group of RY rows (column 0 only hands over its A) are
// laid end to end and cut into warps of 31, the last lane of one repeated as lane
// 0 of the next: tiles of 31 columns leave 15 % of the lanes idle at 160 columns,
// 9 % at 256.  (Lane counts fit an int for any field that fits the GPU.)
// RAW forms the face kappa sums from kappa as the reference does each step
// (the drop-in heat_update); otherwise they are read precomputed, once per
// context: kx[c] = kappa[c] + kappa[c+1], ky[c] = kappa[c] + kappa[c+P],
// kz[c] = kappa[c] + kappa[c+S] -- the same values, fewer additions per point.
//
// Bound: the FP64 pipe (83 % busy, which is all that additions reach), which
// retires about 530 G operations/s, 1/32 of the integer pipes' rate.  A point takes
// 13.7 of them in the reference's order (1 more with a source term, 3.3 more for
// RAW).  Its 3.3 products, and RAW's sums of conductivities, are formed on the
// integer pipes instead (about 40 instructions for a product, 30 for a sum), and so
// is the product with the step factor, but where RAW and a source term leave no
// registers (drop-in 256^3 with source 406 us a step so, 400 with it in FP64;
// without source 2.75 ms for 2.86 at 512^3).  That leaves 9.3 additions.  Where an
// operand is out of their range the lane forms the plane's products again in FP64.
// The differences stay on the FP64 pipe: in integers they must be normalised
// (512^3, GLUP/s: those along z 42 for 48, all 28).
// GLUP/s, all operations in FP64 -> this: context form 160^3 with source 22 -> 38,
// 256^3 30 -> 49.7, 512^3 35.5 -> 52.7; drop-in 256^3 with source 24 -> 41, 512^3
// 28.5 -> 48.
// Blocks are single warps, 12 per SM (168 registers), so that few are left over at
// the end: 160^3 110 us a step for 126 with 4 warps.  Four rows per thread 38.6 for
// 41.6 (drop-in 256^3), two 36 for 48 (512^3).
constexpr int RY = 3;
constexpr int MINB = 12;
template <bool RHS, bool RAW>
constexpr bool kScaled = !(RHS && RAW);

template <bool RHS, bool RAW>
__global__ void __launch_bounds__(32, MINB)
    k_exact_rows(double *__restrict__ un, const double *__restrict__ u,
                 const double *__restrict__ rhs, const double *__restrict__ kap,
                 const double *__restrict__ kx, const double *__restrict__ ky,
                 const double *__restrict__ kz, int nx, int ny, int nz, int P, size_t S,
                 double factor, int kchunk) {
  const int lane = threadIdx.x;
  // Lane 0 repeats the last column of the warp before.
  const int at = blockIdx.x * 31 + lane;
  const int i = at % (nx - 1), j0 = 1 + at / (nx - 1) * RY;
  const int kb = 1 + blockIdx.z * kchunk;
  const int ke = min(kb + kchunk, nz - 1);
  const bool xs = lane >= 1 && i >= 1;
  size_t ro[RY + 2];
#pragma unroll
  for (int t = 0; t < RY + 2; ++t) ro[t] = (size_t)min(j0 - 1 + t, ny - 1) * P + i;
  bool wide = false;  // the factor is out of product()'s range
  const Weight w = weight(factor, wide);
  size_t pl = (size_t)kb * S;
  double uc[RY + 2], kc[RY + 2], F[RY];
  Int wc[RY + 2];     // kc again
  bool below = false;  // a conductivity below zero was seen
#pragma unroll
  for (int t = 0; t < RY + 2; ++t) {
    uc[t] = u[pl + ro[t]];
    kc[t] = RAW ? kap[pl + ro[t]] : 0.0;
    wc[t] = integer(kc[t], below);
  }
#pragma unroll
  for (int r = 0; r < RY; ++r) {
    const size_t q = pl - S + ro[r + 1];
    F[r] = RAW ? flux(__dadd_rn(kc[r + 1], kap[q]), uc[r + 1], u[q])
               : flux(kz[q], uc[r + 1], u[q]);
  }
  for (int k = kb; k < ke; ++k, pl += S) {
    double uu[RY + 2], ku[RY + 2], A[RY], E[RY], G[RY + 1];
    Int wu[RY + 2];
#pragma unroll
    for (int t = 0; t < RY + 2; ++t) {
      uu[t] = u[pl + S + ro[t]];
      ku[t] = RAW ? kap[pl + S + ro[t]] : 0.0;
      wu[t] = integer(ku[t], below);
    }
    // A and E of each row; G[t]: the flux through the face between rows t and t+1
    bool odd = false;
#pragma unroll
    for (int t = 0; t <= RY; ++t)
      G[t] = product(RAW ? sum(wc[t + 1], wc[t], odd) : weight(ky[pl + ro[t]], odd),
                     __dsub_rn(uc[t + 1], uc[t]), odd);
#pragma unroll
    for (int r = 0; r < RY; ++r) {
      const int t = r + 1;
      const size_t q = pl + ro[t];
      A[r] = product(RAW ? sum(integer(kap[q + 1], below), wc[t], odd) : weight(kx[q], odd),
                     __dsub_rn(u[q + 1], uc[t]), odd);
      E[r] = product(RAW ? sum(wu[t], wc[t], odd) : weight(kz[q], odd), __dsub_rn(uu[t], uc[t]),
                     odd);
    }
    if (odd || below) {
#pragma unroll
      for (int t = 0; t <= RY; ++t)
        G[t] = flux(RAW ? __dadd_rn(kc[t + 1], kc[t]) : ky[pl + ro[t]], uc[t + 1], uc[t]);
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        const int t = r + 1;
        const size_t q = pl + ro[t];
        A[r] = flux(RAW ? __dadd_rn(kap[q + 1], kc[t]) : kx[q], u[q + 1], uc[t]);
        E[r] = flux(RAW ? __dadd_rn(ku[t], kc[t]) : kz[q], uu[t], uc[t]);
      }
    }
    double s[RY], ds[RY];
    bool far = wide;
#pragma unroll
    for (int r = 0; r < RY; ++r) {
      const double B = __shfl_up_sync(0xffffffffu, A[r], 1);
      s[r] = walk::net(A[r], B, G[r + 1], G[r], E[r], F[r]);
      ds[r] = kScaled<RHS, RAW> ? product(w, s[r], far) : __dmul_rn(factor, s[r]);
      F[r] = E[r];
    }
    if (kScaled<RHS, RAW> && far) {
      __threadfence_block();  // or the compiler forms these for every lane and selects
#pragma unroll
      for (int r = 0; r < RY; ++r) ds[r] = __dmul_rn(factor, s[r]);
    }
#pragma unroll
    for (int r = 0; r < RY; ++r) {
      const int t = r + 1;
      const size_t q = pl + ro[t];
      if (xs && j0 + r <= ny - 2) un[q] = __dadd_rn(RHS ? __dadd_rn(uc[t], rhs[q]) : uc[t], ds[r]);
    }
#pragma unroll
    for (int t = 0; t < RY + 2; ++t) {
      uc[t] = uu[t];
      kc[t] = ku[t];
      wc[t] = wu[t];
    }
  }
}

template <bool RHS, bool RAW>
void launch_rows(double *u_new, const double *u_old, const double *rhs, const double *kappa,
                 double *const ks[3], const heat_geom &g, double factor, cudaStream_t st) {
  static const long resident = resident_blocks((const void *)k_exact_rows<RHS, RAW>, 32, 0);
  const long lanes = (long)((g.ny - 2 + RY - 1) / RY) * (g.nx - 1);
  const int blocks = (int)((lanes + 30) / 31);
  // Short chunks cost little here (at 192^3 162 us a step with 6 planes, 169 with 16,
  // 198 with 32), and long ones leave SMs idle at the end.
  const int kc = balanced_chunk(blocks, g.nz - 2, resident, 1, 0.4, 10);
  dim3 gr(blocks, 1, (g.nz - 2 + kc - 1) / kc);
  k_exact_rows<RHS, RAW><<<gr, 32, 0, st>>>(
      u_new, u_old, rhs, kappa, ks ? ks[0] : nullptr, ks ? ks[1] : nullptr,
      ks ? ks[2] : nullptr, g.nx, g.ny, g.nz, g.pitch, g.plane, factor, kc);
}

__global__ void k_face_sums(double *__restrict__ kx, double *__restrict__ ky,
                            double *__restrict__ kz, const double *__restrict__ kap,
                            int nx, int ny, int nz, int P, size_t S) {
  // One row (j, k) per block iteration, its points across the threads: no
  // per-point index division.
  const long rows = (long)ny * nz;
  for (long r = blockIdx.x; r < rows; r += gridDim.x)
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    const int j = (int)(r % ny), k = (int)(r / ny);
    const size_t c = (size_t)k * S + (size_t)j * P + i;
    kx[c] = (i + 1 < nx) ? __dadd_rn(kap[c], kap[c + 1]) : 0.0;
    ky[c] = (j + 1 < ny && i < nx) ? __dadd_rn(kap[c], kap[c + P]) : 0.0;
    kz[c] = (k + 1 < nz && i < nx) ? __dadd_rn(kap[c], kap[c + S]) : 0.0;
  }
}


}  // namespace

cudaError_t launch_naive(double *u_new, const double *u_old, const double *rhs,
                         const double *kappa, const heat_geom &g, double factor,
                         cudaStream_t st) {
  dim3 b(8, 8, 8), gr((g.nx + 7) / 8, (g.ny + 7) / 8, (g.nz + 7) / 8);
  if (rhs)
    k_naive<true><<<gr, b, 0, st>>>(u_new, u_old, rhs, kappa, g.nx, g.ny, g.nz, g.pitch,
                                    g.plane, factor);
  else
    k_naive<false><<<gr, b, 0, st>>>(u_new, u_old, rhs, kappa, g.nx, g.ny, g.nz, g.pitch,
                                     g.plane, factor);
  return cudaGetLastError();
}

cudaError_t launch_exact_raw(double *u_new, const double *u_old, const double *rhs,
                             const double *kappa, const heat_geom &g, double factor,
                             cudaStream_t st) {
  if (rhs)
    launch_rows<true, true>(u_new, u_old, rhs, kappa, nullptr, g, factor, st);
  else
    launch_rows<false, true>(u_new, u_old, rhs, kappa, nullptr, g, factor, st);
  return cudaGetLastError();
}

cudaError_t launch_exact_faces(double *u_new, const double *u_old, const double *rhs,
                               double *const ks[3], const heat_geom &g, double factor,
                               cudaStream_t st) {
  if (rhs)
    launch_rows<true, false>(u_new, u_old, rhs, nullptr, ks, g, factor, st);
  else
    launch_rows<false, false>(u_new, u_old, rhs, nullptr, ks, g, factor, st);
  return cudaGetLastError();
}

cudaError_t launch_face_sums(double *const ks[3], const double *kappa, const heat_geom &g,
                             cudaStream_t st) {
  k_face_sums<<<152 * 8, 256, 0, st>>>(ks[0], ks[1], ks[2], kappa, g.nx, g.ny, g.nz,
                                       g.pitch, g.plane);
  return cudaGetLastError();
}

}  // namespace heat
