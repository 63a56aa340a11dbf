// Internal declarations shared by the translation units of libheat.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cmath>
#include <cstddef>
#include <cstdint>

#include "heat.h"

// Device layout of one field: nz planes of ny rows of `pitch` doubles
// (pitch >= nx, a multiple of 4 so every row starts on a 32-byte boundary).
// Padding columns hold zeros and are never read as data.
struct heat_geom {
  int nx, ny, nz;
  int pitch;          // elements per row on the device
  size_t plane;       // pitch * ny
  size_t elems;       // plane * nz
};

struct heat_ctx {
  heat_geom g;
  double h, dt, factor;
  int precision;
  unsigned flags;
  int device;
  cudaStream_t stream;
  bool own_stream;

  // FP64 state: ping-pong fields; cur indexes the current (u_old) one.
  double *u[2];
  int cur;
  double *rhs;              // NULL when the problem has no source term

  // Per-form coefficient planes (only the ones the chosen kernel uses).
  double *kappa;            // raw conductivity (naive kernel; default form, small weights)
  double *ks[3];            // face kappa sums kx, ky, kz (bit-exact kernel)
  double *c0;               // centre weight 1 - sum of face weights (fast, FP64 pipe)
  double *cf[3];            // face weights factor*(kappa_a+kappa_b) (fast, FP64 pipe)
  unsigned long long *kq;   // factor*kappa as fixed-point limbs (default form; NULL: FP64 pipe)

  // FP32C state.
  float *v[2];              // FP32 fields
  uint16_t *carry[2];       // BF16 Kahan carry planes
  float *fcf[3];            // FP32 face weights
  float *frhs;              // FP32 source (NULL when none)

  // Tensor maps of the TMA-staged steps, made once: default FP64 form u0 u1 K rhs,
  // FP32C two-step form v0 v1 carry0 carry1 wx wy wz.
  CUtensorMap maps[7];
  bool have_maps;
  int kchunk;  // planes per block of those steps

  // Device flag a kernel sets when a bounded wait ran out (HEAT_ETIMEOUT).
  int *err;

  // Norm scratch: per-block partial sums, then the final pair.
  double *partials;
  int n_partials;

  long long steps_done;
  long long launches;
};

// ---- kernel launchers (each returns cudaError_t of the launch) ----------
namespace heat {

#ifdef __CUDACC__
// Face weight factor * (ka + kb) and centre weight
// 1 - (((((e + w) + n) + s) + u) + d) of the default FP64 form, every operation
// rounded on its own (no fused multiply-add), so every kernel that forms them
// gets the same bits.
__device__ __forceinline__ double fw(double factor, double ka, double kb) {
  return __dmul_rn(factor, __dadd_rn(ka, kb));
}
__device__ __forceinline__ double centre(double e, double w, double n, double s, double u,
                                         double d) {
  return __dsub_rn(1.0, __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(e, w), n), s), u), d));
}
#endif

#ifdef __CUDACC__
// A TMA-staged step kernel begins with chain(): it lets the next launch of its
// stream start (blocks set up, waiting in their own chain()) and waits until the
// launch before it is complete and its results visible.  Nothing may touch a
// field before it.  The L1 caches keep their read-only lines from one chained
// launch to the next, so such a kernel reads global memory by TMA or __ldcg only:
// the column-walk kernels (const __restrict__ fields) and the batch kernels
// (tables, which the host rewrites) have plain launches, before which chain()
// does nothing.
__device__ __forceinline__ void chain() {
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}

// Launches a kernel that begins with chain(), so that it may start before the
// kernel ahead of it on the stream ends.  Launches after it that are not made
// through here still wait for all of it.
template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                           cudaStream_t st, A... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
#endif

constexpr int kNormBlocks = 152 * 4;   // partial-sum blocks of the norm pass

// Bound of every device-side mbarrier wait in the TMA kernels (try_wait
// attempts of about 4 us); a wait that runs out sets the context's error flag and
// the launch returns with its outputs unwritten.  Blocks that start with the flag
// set leave at once, so all that is queued behind a failure ends within a wait.
constexpr unsigned kWaitLimit = 1u << 22;
// The same in the table kernels: 65 ms.  Their loads go by tensor maps in device
// memory, and a wrong one is a load that never completes.
constexpr unsigned kTableWaitLimit = 1u << 14;

// Planes per block for a launch of (tile_x x tile_y)-column tiles over the
// grid's interior: enough z-chunks that tiles x chunks reaches `want` blocks
// (16 per SM of GB300's 152 by default), at least 8 planes each.
inline int plane_chunk(const heat_geom &g, int tile_x, int tile_y, long want = 152L * 16) {
  const long tiles =
      (long)((g.nx - 2 + tile_x - 1) / tile_x) * ((g.ny - 2 + tile_y - 1) / tile_y);
  const long chunks = (want + tiles - 1) / tiles;
  const int interior = g.nz - 2;
  int kc = (int)((interior + chunks - 1) / chunks);
  if (kc < 8) kc = 8;
  if (kc > interior) kc = interior;
  return kc;
}

// Blocks of `kernel` resident on the current GPU at once: its occupancy per
// SM at `threads` threads and `smem` bytes of dynamic shared memory per block,
// times the SM count; 0 when the runtime cannot say (heat_abi.cpp).  The
// launchers look it up once per process (one GPU model per process).
long resident_blocks(const void *kernel, int threads, size_t smem);

// Planes per block for a launch of (tile_x x tile_y)-column tiles whose blocks
// run `resident` at a time: enough z-chunks that the launch spans about
// `waves` waves of resident blocks, so the last wave, which the GPU may run
// partly empty, is a small share of it; at least `min_planes` planes per chunk
// (each chunk re-reads its halo planes and refills its pipeline) unless that
// would leave fewer than two waves.  Used by the column walks: at 512^3 the FP64-pipe
// one runs 85.0 GLUP/s so (79.2 with plane_chunk), the FP32C one 210.6 (188.0).  Falls
// back to plane_chunk when `resident` is unknown.
inline int wave_chunk(const heat_geom &g, int tile_x, int tile_y, long resident,
                      long waves = 24, int min_planes = 16, int fill_planes = 8) {
  if (resident <= 0) return plane_chunk(g, tile_x, tile_y);
  const long tiles =
      (long)((g.nx - 2 + tile_x - 1) / tile_x) * ((g.ny - 2 + tile_y - 1) / tile_y);
  const int interior = g.nz - 2;
  long chunks = (resident * waves + tiles - 1) / tiles;
  const long max_chunks = interior / min_planes > 1 ? interior / min_planes : 1;
  if (chunks > max_chunks) chunks = max_chunks;
  // A grid too small for `waves` waves at that depth still gets two waves of
  // blocks where chunks of `fill_planes` planes allow it, so it does not leave
  // SMs idle.
  long fill = (2 * resident + tiles - 1) / tiles;
  if (fill > interior / fill_planes) fill = interior / fill_planes;
  if (chunks < fill) chunks = fill;
  if (chunks < 1) chunks = 1;
  return (int)((interior + chunks - 1) / chunks);
}

// Planes per block for a launch of `tiles` tiles over `interior` planes whose
// blocks run `resident` at a time: the chunk count with the least estimated
// time.  A round of blocks takes (planes + overhead) plane times; `alone` is a
// plane's time with one block on an SM as a fraction of its time on a full one
// (latency keeps it from falling with the load), between which it rises steeply
// at first (k_fx: 0.53, 0.88, 0.94, 1 for 1 to 4 blocks).  At most `most` planes:
// few long rounds end less evenly than this counts on; more only where a launch
// could not have that many chunks.  Against the chunk that measured best of 19 it costs 2 to 8 % on
// grids from 40 x 33 x 28 to 512^3.
constexpr int kMaxGridZ = 65535;  // most blocks along z of a launch
inline int balanced_chunk(long tiles, int interior, long resident, int overhead, double alone,
                          int most) {
  const int least = (interior + kMaxGridZ - 1) / kMaxGridZ;
  if (most < least) most = least;
  if (resident <= 0) return interior < most ? interior : most;
  const long per_sm = (resident + 151) / 152;
  double best = 0;
  int best_kc = 0;
  for (int most_kc = interior < most ? interior : most; most_kc >= least; --most_kc) {
    const int chunks = (interior + most_kc - 1) / most_kc;
    const int kc = (interior + chunks - 1) / chunks;
    const long blocks = tiles * chunks;
    const long rest = (blocks % resident + 151) / 152;  // blocks per SM in the last round
    double rounds = (double)(blocks / resident);
    if (rest)
      rounds += alone + (1.0 - alone) * std::sqrt((double)(rest - 1) / (per_sm > 1 ? per_sm - 1 : 1));
    const double cost = rounds * (kc + overhead);
    if (best_kc == 0 || cost < best) {
      best = cost;
      best_kc = kc;
    }
  }
  return best_kc;
}

// Sheets of a few rows, which the TMA-staged kernels' tiles (16 and 20 rows high) would
// leave mostly empty, step with the column walks instead, where the sheet is large
// enough that a step is not all launch.  us a step, walk and tiles: default form (two
// rows at most) 4096 x 4 x 2048 231 and 438, 512 x 4 x 512 15.0 and 17.4, but 256 x 4 x
// 256 8.3 and 7.5, and three rows of 1024 x 1024 64 and 59; FP32C (eight rows at most)
// 1024 x 10 x 1024 50 and 54, 512 x 3 x 512 10.3 and 14.6, but 256 x 10 x 256 7.7 and
// 6.2, and ten rows of 1024 x 1024 72 and 54.
inline bool thin_sheet(const heat_geom &g, int rows) {
  return g.ny - 2 <= rows && (long long)(g.nx - 2) * (g.nz - 2) >= 200000;
}
constexpr int kThinRowsFp64 = 2, kThinRowsFp32c = 8;

// heat_fp64_exact.cu (compiled with --fmad=false)
cudaError_t launch_exact_raw(double *u_new, const double *u_old, const double *rhs,
                             const double *kappa, const heat_geom &g, double factor,
                             cudaStream_t st);
cudaError_t launch_exact_faces(double *u_new, const double *u_old, const double *rhs,
                               double *const ks[3], const heat_geom &g, double factor,
                               cudaStream_t st);
cudaError_t launch_naive(double *u_new, const double *u_old, const double *rhs,
                         const double *kappa, const heat_geom &g, double factor,
                         cudaStream_t st);
cudaError_t launch_face_sums(double *const ks[3], const double *kappa, const heat_geom &g,
                             cudaStream_t st);

// heat_fp64_fast.cu
cudaError_t launch_fast_coeffs(double *c0, double *const cf[3], const double *kappa,
                               const heat_geom &g, double factor, cudaStream_t st);
cudaError_t launch_fast(double *u_new, const double *u_old, const double *rhs,
                        const double *c0, double *const cf[3], const heat_geom &g,
                        cudaStream_t st);

// heat_fp64_weights.cu: the default form's fixed-point weights; bad[0] (zeroed
// by the caller) is set when the form cannot represent the problem.
cudaError_t launch_kq_setup(unsigned long long *K, int *bad, const double *kappa,
                            const heat_geom &g, double factor, cudaStream_t st);

// heat_fp64_fx.cu: one step of the default form (fixed point, TMA-staged) of
// context c from buffer `cur`.  encode_fx_maps fills m with the maps of a
// field pair, its weights and source term (NULL: none).
bool fx_usable(bool rhs);
int fx_chunk(const heat_geom &g, bool rhs);
bool encode_fx_maps(CUtensorMap *m, double *const u[2], const unsigned long long *K,
                    const double *rhs, const heat_geom &g);
cudaError_t launch_fx(const heat_ctx *c, int cur, cudaStream_t st,
                      unsigned wait_limit = kWaitLimit);
// n steps of context c from buffer `cur` on stream st with its own
// single-grid kernels (two steps per launch where its form has them); the
// context's bookkeeping is untouched.  ctx_flips gives the parity of buffer
// swaps those n steps make (a two-step launch swaps once).
cudaError_t enqueue_ctx_steps(heat_ctx *c, int cur, long long n, cudaStream_t st,
                              long long *launches);
int ctx_flips(const heat_ctx *c, long long n);
// One step of context c from buffer `cur` with its single-grid one-step kernel.
cudaError_t enqueue_one_step(heat_ctx *c, int cur, cudaStream_t st, long long *launches);

// heat_fp32c.cu
cudaError_t launch_fp32c(float *v_new, uint16_t *c_new, const float *v, const uint16_t *cr,
                         float *const w[3], const float *rhs, const heat_geom &g,
                         cudaStream_t st);
cudaError_t launch_split(float *v, uint16_t *cr, const double *u, size_t total, cudaStream_t st);
cudaError_t launch_widen(double *u, const float *v, const uint16_t *cr, size_t total,
                         cudaStream_t st);
cudaError_t launch_f32_weights(float *const w[3], const double *kappa, const heat_geom &g,
                               double factor, cudaStream_t st);
cudaError_t launch_to_f32(float *o, const double *a, size_t total, cudaStream_t st);

// heat_fp32c_tma.cu: two steps per launch (temporal blocking, TMA staging) of
// context c from buffer `cur`.  wait_limit bounds every mbarrier wait of the
// launch (kWaitLimit in product use; smaller only to exercise the failure path).
bool encode_fp32c_maps(CUtensorMap *m, float *const v[2], uint16_t *const cr[2],
                       float *const w[3], const heat_geom &g);
int fp32c_tb2_chunk(const heat_geom &g);
cudaError_t launch_fp32c_tb2(const heat_ctx *c, int cur, cudaStream_t st,
                             unsigned wait_limit = kWaitLimit);
// Whether a context steps with launch_fp32c_tb2.
bool two_step_form(const heat_ctx *c);
// HEAT_ETIMEOUT if a kernel of context c reported a bounded wait running out
// (the flag is cleared once reported), else HEAT_OK.  Synchronises c's stream.
int check_err(heat_ctx *c);
// Record a failed CUDA call for heat_strerror() and return HEAT_ECUDA.
int cuda_fail(cudaError_t e, const char *what);

// heat_reduce.cu
cudaError_t launch_norm_f64(const double *u, const heat_geom &g, double *partials,
                            int nblocks, cudaStream_t st);
// Norm of the FP32C state u = v - c (widened to FP64 per point).
cudaError_t launch_norm_f32c(const float *v, const uint16_t *cr, const heat_geom &g,
                             double *partials, int nblocks, cudaStream_t st);
// sum (a-b)^2, sum b^2 and max |a-b| of two FP64 fields of one geometry;
// partials needs 3*nblocks+3 doubles, results at partials[3*nblocks..].
cudaError_t launch_diff_f64(const double *a, const double *b, const heat_geom &g,
                            double *partials, int nblocks, cudaStream_t st);

}  // namespace heat
