// Per-column "walks" shared by the single-grid kernels and the batched
// persistent kernel: each walks one (i, j) column of a grid over planes
// [kb, ke), z-neighbours held in registers, and writes the new values.  The
// same code runs alone and in a batch, so a grid's results do not depend on
// how it was launched.

#pragma once

#include <cuda_bf16.h>
#include <cstdint>

namespace heat {
namespace walk {
namespace {

// ---- bit-exact FP64 (reference operation order, every operation rounded) ----
__device__ __forceinline__ double flux(double ksum, double ub, double ua) {
  return __dmul_rn(ksum, __dsub_rn(ub, ua));
}

// The sum of the face fluxes in the reference's order.
__device__ __forceinline__ double net(double A, double B, double C, double D, double E, double F) {
  return __dsub_rn(__dadd_rn(__dsub_rn(__dadd_rn(__dsub_rn(A, B), C), D), E), F);
}

// base is u + rhs (or u alone when the problem has no source term: u + 0.0
// equals u for every value but -0.0, which these fields never hold).
__device__ __forceinline__ double combine(double base, double factor, double A, double B,
                                          double C, double D, double E, double F) {
  return __dadd_rn(base, __dmul_rn(factor, net(A, B, C, D, E, F)));
}

template <bool RHS>
__device__ __forceinline__ void walk_exact_faces(double *__restrict__ un,
                                                 const double *__restrict__ u,
                                                 const double *__restrict__ rhs,
                                                 const double *__restrict__ kx,
                                                 const double *__restrict__ ky,
                                                 const double *__restrict__ kz, int P,
                                                 size_t S, size_t c, int kb, int ke,
                                                 double factor) {
  double uc = u[c];
  double F = flux(kz[c - S], uc, u[c - S]);
  for (int k = kb; k < ke; ++k, c += S) {
    double uu = u[c + S];
    double A = flux(kx[c], u[c + 1], uc);
    double B = flux(kx[c - 1], uc, u[c - 1]);
    double C = flux(ky[c], u[c + P], uc);
    double D = flux(ky[c - P], uc, u[c - P]);
    double E = flux(kz[c], uu, uc);
    un[c] = combine(RHS ? __dadd_rn(uc, rhs[c]) : uc, factor, A, B, C, D, E, F);
    F = E;
    uc = uu;
  }
}

// Column state of the FP64-pipe walk (precomputed double weights, 7 FMA per
// point).  The plane's loads are issued one step ahead, so they overlap the
// arithmetic.
template <bool RHS>
struct HwCol {
  size_t c;
  double ud, uc, wd;
  double nu, nwu, nc0, nr, nxe, nxw, nyn, nys, ne, nw, nn, ns;

  __device__ __forceinline__ void fetch(const double *__restrict__ u,
                                        const double *__restrict__ rhs,
                                        const double *__restrict__ c0,
                                        const double *__restrict__ cx,
                                        const double *__restrict__ cy,
                                        const double *__restrict__ cz, int P, size_t S,
                                        size_t q) {
    nu = u[q + S];
    nwu = cz[q];
    nc0 = c0[q];
    nr = RHS ? rhs[q] : 0.0;
    nxe = cx[q];
    nxw = cx[q - 1];
    nyn = cy[q];
    nys = cy[q - P];
    ne = u[q + 1];
    nw = u[q - 1];
    nn = u[q + P];
    ns = u[q - P];
  }

  __device__ __forceinline__ void start(const double *__restrict__ u,
                                        const double *__restrict__ rhs,
                                        const double *__restrict__ c0,
                                        const double *__restrict__ cx,
                                        const double *__restrict__ cy,
                                        const double *__restrict__ cz, int P, size_t S,
                                        size_t c_) {
    c = c_;
    ud = u[c - S];
    uc = u[c];
    wd = cz[c - S];
    fetch(u, rhs, c0, cx, cy, cz, P, S, c);
  }

  __device__ __forceinline__ void step(double *__restrict__ un, const double *__restrict__ u,
                                       const double *__restrict__ rhs,
                                       const double *__restrict__ c0,
                                       const double *__restrict__ cx,
                                       const double *__restrict__ cy,
                                       const double *__restrict__ cz, int P, size_t S,
                                       bool more) {
    const double uu = nu, wu = nwu, w0 = nc0, r = nr, xe = nxe, xw = nxw, yn = nyn, ys = nys;
    const double ue = ne, uw = nw, un_ = nn, us = ns;
    if (more) fetch(u, rhs, c0, cx, cy, cz, P, S, c + S);
    double acc = RHS ? fma(w0, uc, r) : w0 * uc;
    acc = fma(xe, ue, acc);
    acc = fma(xw, uw, acc);
    acc = fma(yn, un_, acc);
    acc = fma(ys, us, acc);
    acc = fma(wu, uu, acc);
    acc = fma(wd, ud, acc);
    un[c] = acc;
    ud = uc;
    uc = uu;
    wd = wu;
    c += S;
  }
};

// The FP64-pipe walk over one (i, j) column, planes [kb, ke).
template <bool RHS>
__device__ __forceinline__ void walk_hw(double *__restrict__ un, const double *__restrict__ u,
                                        const double *__restrict__ rhs,
                                        const double *__restrict__ c0,
                                        const double *__restrict__ cx,
                                        const double *__restrict__ cy,
                                        const double *__restrict__ cz, int P, size_t S,
                                        size_t c, int kb, int ke) {
  HwCol<RHS> col;
  col.start(u, rhs, c0, cx, cy, cz, P, S, c);
  for (int k = kb; k < ke; ++k) col.step(un, u, rhs, c0, cx, cy, cz, P, S, k + 1 < ke);
}

// ---- FP32-compensated form ----
__device__ __forceinline__ float bf2f(uint16_t b) {
  return __uint_as_float(((unsigned)b) << 16);
}
__device__ __forceinline__ uint16_t f2bf(float x) {
  __nv_bfloat16 h = __float2bfloat16_rn(x);
  return *reinterpret_cast<uint16_t *>(&h);
}

template <bool RHS>
__device__ __forceinline__ void walk_fp32c(float *__restrict__ vn, uint16_t *__restrict__ cn,
                                           const float *__restrict__ v,
                                           const uint16_t *__restrict__ cr,
                                           const float *__restrict__ wx,
                                           const float *__restrict__ wy,
                                           const float *__restrict__ wz,
                                           const float *__restrict__ rhs, int P, size_t S,
                                           size_t c, int kb, int ke) {
  float vd = v[c - S], vc = v[c];
  float wd = wz[c - S];
  // The plane's loads are issued one iteration ahead (the walk is bound by
  // memory latency, not arithmetic).
  float nu = v[c + S], nwz = wz[c], ne = v[c + 1], nw = v[c - 1], nn = v[c + P], ns = v[c - P];
  float nwx = wx[c], nwxm = wx[c - 1], nwy = wy[c], nwym = wy[c - P];
  uint16_t ncr = cr[c];
  float nr = RHS ? rhs[c] : 0.0f;
  for (int k = kb; k < ke; ++k, c += S) {
    const float vu = nu, wu = nwz, ve = ne, vw = nw, vn_ = nn, vs = ns;
    const float w_e = nwx, w_w = nwxm, w_n = nwy, w_s = nwym, r = nr;
    const uint16_t cc0 = ncr;
    if (k + 1 < ke) {
      const size_t q = c + S;
      nu = v[q + S];
      nwz = wz[q];
      ne = v[q + 1];
      nw = v[q - 1];
      nn = v[q + P];
      ns = v[q - P];
      nwx = wx[q];
      nwxm = wx[q - 1];
      nwy = wy[q];
      nwym = wy[q - P];
      ncr = cr[q];
      if (RHS) nr = rhs[q];
    }
    float d = r;
    d = fmaf(w_e, ve - vc, d);
    d = fmaf(w_w, vw - vc, d);
    d = fmaf(w_n, vn_ - vc, d);
    d = fmaf(w_s, vs - vc, d);
    d = fmaf(wu, vu - vc, d);
    d = fmaf(wd, vd - vc, d);
    const float y = __fsub_rn(d, bf2f(cc0));
    const float t = __fadd_rn(vc, y);
    const float cc = __fsub_rn(__fsub_rn(t, vc), y);
    vn[c] = t;
    cn[c] = f2bf(cc);
    vd = vc;
    vc = vu;
    wd = wu;
  }
}

}  // namespace
}  // namespace walk
}  // namespace heat
