// FP32-compensated form, two time steps per launch (temporal blocking), with
// plane tiles staged into shared memory by TMA.
//
// A block owns a (32 x 20) tile of output columns and walks a chunk of planes;
// it has one thread per pair of neighbouring columns of the tile plus a 1-point
// halo (17 pairs by 22 rows: 374 threads in 12 warps, three on each of the SM's
// four schedulers), and computes both with GB300's packed FP32 operations.
// For every plane p the block's thread 0 issues TMA 3-D box loads
// (cp.async.bulk.tensor) of the five input arrays -- v, carry, wx, wy, wz --
// covering the tile plus a 2-point halo into one slot of a 4-deep shared
// memory ring, completing on that slot's mbarrier; loads run two planes ahead
// of use.  Each iteration k then
//   1. computes step t+1 on plane k+1 over the tile plus a 1-point halo
//      (34 x 22 points) from ring planes k, k+1, k+2 into a 3-plane ring of
//      intermediate values, and
//   2. computes step t+2 on plane k-1 over the tile from intermediate planes
//      k-2, k-1, k and writes it to global memory.
// Running step t+2 one plane behind step t+1 leaves one block barrier per
// plane (it publishes the landed input plane and the previous iteration's
// intermediate plane together), and makes the two steps of an iteration
// independent of each other.
// Global traffic per two updates: the five input arrays read once (plus the
// halo, mostly served by L2) and v, carry written once -- about half of two
// single steps.  The per-point arithmetic is exactly the single-step column
// walk's (walk_fp32c: same operations, same order, the intermediate carry
// rounded to BF16 as the single step stores it), so two steps here are
// bit-identical to two single steps.  Points on the grid boundary keep their
// values at both levels.
//
// Bound: issue and latency between the barriers (24 warps an SM, issue 52 % busy at
// 400^3, shared-memory reads the first stall).  512^3: 375 GLUP/s, where one thread per point in 20 warps ran 331.
// Measured and not kept at 512^3: 16 rows (10 warps of pairs, which load the
// schedulers 3 : 3 : 2 : 2) 327, three blocks of them per SM at 64 registers 355;
// 13 rows in 8 warps, three blocks per SM, 357; 28 rows in 16 warps 319; two
// planes per barrier with a 5-deep ring 346 (20 rows); the steps under their own
// conditions instead of in one straight line 313 for 326 (16 rows).
//
// Every mbarrier wait is bounded: if a load does not complete within the
// limit the block records the failure in *err, waits (bounded) for its other
// loads in flight, and returns; the host reports HEAT_ETIMEOUT.

#include <cuda.h>

#include "heat_batch_internal.h"
#include "heat_internal.h"
#include "heat_tma.cuh"
#include "heat_walk.cuh"

namespace heat {
namespace {

constexpr int OX = 32, OY = 20;          // output tile
constexpr int BXF = 40, BXC = 48, BY = OY + 4;  // TMA boxes (float arrays, BF16 carry)
constexpr int LP = (OX + 2) / 2, L1Y = OY + 2;  // step-(t+1) region: pairs by rows
constexpr int NT = (LP * L1Y + 31) / 32 * 32;   // one thread per pair
constexpr int V1X = 2 * LP + 2;                 // row of the intermediate planes
constexpr int R = 4;                     // ring depth (planes)
static_assert((R & (R - 1)) == 0, "slot index p & (R - 1) needs R a power of two");

constexpr int kPlaneF = BXF * BY;        // floats per float-array plane tile
constexpr int kPlaneC = BXC * BY;        // BF16 per carry plane tile
constexpr unsigned kSlotBytes = 4u * kPlaneF * 4u + 2u * kPlaneC;  // v, wx, wy, wz + carry
// A TMA tile copy writes shared memory from a 128-byte aligned address, so
// each array of a slot starts on a 128-byte boundary: arrays are strided by
// their box size rounded up to 128 bytes (the copies still move box bytes).
constexpr int kStrideF = (kPlaneF * 4 + 127) / 128 * 128 / 4;
constexpr int kStrideC = (kPlaneC * 2 + 127) / 128 * 128 / 2;
static_assert((kStrideF * 4) % 128 == 0 && (kStrideC * 2) % 128 == 0,
              "slot arrays must start on 128-byte boundaries");

struct __align__(128) Slot {
  float v[kStrideF];
  float wx[kStrideF];
  float wy[kStrideF];
  float wz[kStrideF];
  uint16_t c[kStrideC];
};
static_assert(sizeof(Slot) % 128 == 0, "ring slots must start on 128-byte boundaries");

struct Smem {
  Slot ring[R];
  __align__(8) float v1[3][V1X * (L1Y + 2)];  // a spare row at either end
  unsigned long long bar[R];
};

using tma::mbar_expect;
using tma::mbar_init;
using tma::mbar_wait;
using tma::smem_u32;

__device__ __forceinline__ void tma_load3(void *dst, const CUtensorMap *map, int x, int y, int z,
                                          unsigned long long *bar) {
  tma::load3(dst, map, x, y, z, bar);
}

struct Maps {
  CUtensorMap v, c, wx, wy, wz;
};

// Where a tile finds its five tensor maps: the single-grid kernel's
// __grid_constant__ parameters, or seven maps per grid in device memory for
// the batch table (buffer `src` of v and carry, then wx, wy, wz).
struct ParamMaps {
  static constexpr bool kInMemory = false;
  static constexpr unsigned kLimit = kWaitLimit;
  const Maps &in;
  __device__ __forceinline__ const CUtensorMap *v() const { return &in.v; }
  __device__ __forceinline__ const CUtensorMap *c() const { return &in.c; }
  __device__ __forceinline__ const CUtensorMap *wx() const { return &in.wx; }
  __device__ __forceinline__ const CUtensorMap *wy() const { return &in.wy; }
  __device__ __forceinline__ const CUtensorMap *wz() const { return &in.wz; }
};
struct TableMaps {
  static constexpr bool kInMemory = true;
  static constexpr unsigned kLimit = kTableWaitLimit;
  const CUtensorMap *tm;
  int src;
  __device__ __forceinline__ const CUtensorMap *v() const { return &tm[src]; }
  __device__ __forceinline__ const CUtensorMap *c() const { return &tm[2 + src]; }
  __device__ __forceinline__ const CUtensorMap *wx() const { return &tm[4]; }
  __device__ __forceinline__ const CUtensorMap *wy() const { return &tm[5]; }
  __device__ __forceinline__ const CUtensorMap *wz() const { return &tm[6]; }
};

// Two FP32 values side by side in a 64-bit register, and GB300's packed FP32
// operations on them: each half rounds as the scalar operation does.
typedef unsigned long long f2;

__device__ __forceinline__ f2 pair(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo(f2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi(f2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a - b: -1 * b is exact, so one rounding, as in the scalar subtraction
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, 0xbf800000bf800000ull, a); }
__device__ __forceinline__ f2 ld2(const float *p) { return *reinterpret_cast<const f2 *>(p); }
// BF16 pair to and from FP32
__device__ __forceinline__ f2 wide(unsigned c) {
  return pair(__uint_as_float(c << 16), __uint_as_float(c & 0xffff0000u));
}
__device__ __forceinline__ unsigned bf16(f2 a) {
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi(a)), "f"(lo(a)));
  return r;
}

// Face weights of a pair at one plane: wx[c], wx[c+1]; wx[c-1]; wy[c]; wy[c-P];
// wz[c].
struct W {
  f2 x;
  float xw;
  f2 y, ym, z;
};

// Kahan step of a pair: centre c, in-plane neighbours (we, ee: the scalars west
// and east of the pair), planes above and below, carry cc.  The operations and
// their order are walk_fp32c's.
__device__ __forceinline__ f2 kahan(const W &w, f2 wzm, f2 c, float ww, float ee, f2 n, f2 s, f2 up,
                                    f2 dn, f2 cc, f2 &carry) {
  f2 d = fma2(w.x, sub2(pair(hi(c), ee), c), 0ull);
  d = fma2(pair(w.xw, lo(w.x)), sub2(pair(ww, lo(c)), c), d);
  d = fma2(w.y, sub2(n, c), d);
  d = fma2(w.ym, sub2(s, c), d);
  d = fma2(w.z, sub2(up, c), d);
  d = fma2(wzm, sub2(dn, c), d);
  const f2 y = sub2(d, cc);
  const f2 t = add2(c, y);
  carry = sub2(sub2(t, c), y);
  return t;
}

// Two steps over one (32 x 20)-column tile with origin (x0, y0), planes
// [kb, ke), of a field whose five input arrays the maps describe.  Writes vn
// / cn.  When a bounded wait runs out it sets *err and returns once its own
// loads in flight have landed.
template <class M>
__device__ __forceinline__ void tb2_tile(const M &maps, float *__restrict__ vn,
                                         uint16_t *__restrict__ cn, int x0, int y0, int nx,
                                         int ny, int nz, int P, size_t S, int kb, int ke,
                                         int *__restrict__ err, unsigned wait_limit) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  const int tid = threadIdx.x;
  const int X0 = x0 - 5, X0c = x0 - 9, Y0 = y0 - 2;  // box origins (X0 % 4 == 0, X0c % 8 == 0)
  const int pmin = max(kb - 2, 0), pmax = min(ke + 1, nz - 1);

  if (tid == 0) {
    for (int s = 0; s < R; ++s) mbar_init(&sm.bar[s]);
    tma::mbar_init_fence();
  }
  chain();

  // Every warp waits on the mbarriers itself (warp 0 alone, handing the planes
  // on through the block barrier: 319 GLUP/s for 335 at 384^3); thread 0 issues
  // the TMA.
  unsigned pending = 0, phase = 0;
  bool failed = false;
  auto issue = [&](int p) {
    if (p < pmin || p > pmax) return;
    const int s = p & (R - 1);
    pending |= 1u << s;
    if (tid != 0) return;
    Slot &sl = sm.ring[s];
    unsigned long long *b = &sm.bar[s];
    tma::fence_proxy_async();
    mbar_expect(b, kSlotBytes);
    tma_load3(sl.v, maps.v(), X0, Y0, p, b);
    tma_load3(sl.wx, maps.wx(), X0, Y0, p, b);
    tma_load3(sl.wy, maps.wy(), X0, Y0, p, b);
    tma_load3(sl.wz, maps.wz(), X0, Y0, p, b);
    tma_load3(sl.c, maps.c(), X0c, Y0, p, b);
  };
  auto wait_plane = [&](int p) {
    if (p < pmin || p > pmax || failed) return;
    const int s = p & (R - 1);
    if (!mbar_wait(&sm.bar[s], (phase >> s) & 1u, wait_limit)) {
      failed = true;
      return;
    }
    phase ^= 1u << s;
    pending &= ~(1u << s);
  };

  // The flag is read before the first loads where a wrong map could be what set it, else
  // beside them by another warp, and looked at with the first planes.
  bool stop = tid == (M::kInMemory ? 0 : NT - 1) && tma::gave_up(err);
  if (M::kInMemory) {
    if (__syncthreads_or(stop)) return;
    stop = false;
  }
  for (int p = kb - 2; p <= kb + 1; ++p) issue(p);
  if (!M::kInMemory) __syncthreads();
  // Before the block's shared memory goes its own loads in flight must have landed
  // (each wait bounded).
  auto drain = [&] {
    for (int s = 0; s < R; ++s)
      if (pending & (1u << s)) mbar_wait(&sm.bar[s], (phase >> s) & 1u, M::kLimit);
  };

  // This thread's step-(t+1) points: columns gx, gx + 1 (gx even) of row gy,
  // pair lp and row ly of the (17 x 22) region, and their shared-memory offsets.
  // Those with 1 <= column <= 32 and 1 <= ly <= 20 of the region are output
  // points.  Like the single-step walk, each thread carries its own columns
  // along z in registers: the centre values of the input planes, the step-(t+1)
  // values it computed, and the face weights it already loaded; only neighbours
  // come from shared memory.
  const int lp = tid % LP;
  const bool l1_ok = tid < LP * L1Y;
  const int ly = l1_ok ? tid / LP : 0;  // threads past the region walk its first row and store nothing
  const int gx = x0 - 1 + 2 * lp, gy = y0 - 1 + ly;
  const int o = (ly + 1) * BXF + 2 * lp + 4;      // float box offset
  const int oc = (ly + 1) * BXC + 2 * lp + 8;     // carry box offset
  const int o1 = (ly + 1) * V1X + 2 * lp;         // intermediate plane offset
  const bool edge_y = gy <= 0 || gy >= ny - 1;
  const bool edge0 = edge_y || gx <= 0 || gx >= nx - 1, edge1 = edge_y || gx + 1 >= nx - 1;
  // Whether the tile's step-(t+1) region reaches the grid's boundary in x or y.
  const bool edge_tile = x0 == 1 || y0 == 1 || x0 + OX >= nx - 1 || y0 + OY >= ny - 1;
  const bool out_y = l1_ok && ly >= 1 && ly <= OY && gy < ny - 1;
  const bool out0 = out_y && lp > 0 && gx < nx - 1, out1 = out_y && lp < LP - 1 && gx + 1 < nx - 1;

  // Step t+1 on plane p at this thread's points from centre values vm, v0, vp
  // (planes p-1, p, p+1) and wz at plane p-1; returns the new values and
  // carries and the plane's weights.
  auto level1 = [&](int p, f2 vm, f2 v0, f2 vp, f2 wzm, W &wp, f2 &t1, f2 &c1) {
    const Slot &cur = sm.ring[p & (R - 1)];
    wp.x = ld2(&cur.wx[o]);
    wp.xw = cur.wx[o - 1];
    wp.y = ld2(&cur.wy[o]);
    wp.ym = ld2(&cur.wy[o - BXF]);
    wp.z = ld2(&cur.wz[o]);
    const f2 cc0 = wide(*reinterpret_cast<const unsigned *>(&cur.c[oc]));
    f2 c;
    const f2 t = kahan(wp, wzm, v0, cur.v[o - 1], cur.v[o + 2], ld2(&cur.v[o + BXF]),
                       ld2(&cur.v[o - BXF]), vp, vm, cc0, c);
    t1 = t;
    c1 = wide(bf16(c));
    const bool z = p == 0 || p == nz - 1;
    if (edge_tile || z) {  // the same for the whole block
      t1 = pair(edge0 || z ? lo(v0) : lo(t1), edge1 || z ? hi(v0) : hi(t1));
      c1 = pair(edge0 || z ? lo(cc0) : lo(c1), edge1 || z ? hi(cc0) : hi(c1));
    }
  };

  // Prologue: intermediate planes kb-1 and kb.  A failed wait stops the whole
  // block (the decision is made block-wide).
  wait_plane(kb - 2);
  wait_plane(kb - 1);
  wait_plane(kb);
  wait_plane(kb + 1);
  failed = __syncthreads_or(failed || stop);
  // Level-1 window: v(p-1), v(p), wz(p-1) for the next plane p to compute.
  f2 vm = 0, v0 = 0, wzm = 0;
  // Level-2 window at the top of iteration k: own step-(t+1) values at planes
  // k-2, k-1, k, the carries at k-1, k, the weights at k-1, k and wz at k-2.
  f2 l1a = 0, l1b = 0, l1cc = 0;
  f2 c1b = 0, c1cc = 0;
  W wb{}, wcc{};
  f2 wza = 0;
  if (!failed && l1_ok) {
    if (kb - 2 >= 0) {
      vm = ld2(&sm.ring[(kb - 2) & (R - 1)].v[o]);
      wzm = ld2(&sm.ring[(kb - 2) & (R - 1)].wz[o]);
    }
    v0 = ld2(&sm.ring[(kb - 1) & (R - 1)].v[o]);
    f2 vp = ld2(&sm.ring[kb & (R - 1)].v[o]);
    level1(kb - 1, vm, v0, vp, wzm, wb, l1b, c1b);
    *reinterpret_cast<f2 *>(&sm.v1[(kb - 1) % 3][o1]) = l1b;
    vm = v0;
    v0 = vp;
    wzm = wb.z;
    vp = ld2(&sm.ring[(kb + 1) & (R - 1)].v[o]);
    level1(kb, vm, v0, vp, wzm, wcc, l1cc, c1cc);
    *reinterpret_cast<f2 *>(&sm.v1[kb % 3][o1]) = l1cc;
    vm = v0;
    v0 = vp;
    wzm = wcc.z;
  }
  // The prologue's reads of planes kb-2 and kb-1 are done: their slots take
  // planes kb+2 and kb+3.
  __syncthreads();
  if (!failed) {
    issue(kb + 2);
    issue(kb + 3);
  }

  // Step t+2 runs one plane behind step t+1: iteration k computes step t+1 on
  // plane k+1 and step t+2 on plane k-1, so the one barrier at the top of an
  // iteration publishes both the landed plane k+2 and the previous
  // iteration's step-(t+1) plane k, and retires ring slot k mod R and
  // intermediate slot (k+1) mod 3 for reuse.  Iteration kb writes no output
  // (plane kb-1 is outside the chunk); iteration ke computes no step t+1.
  // Intermediate slots of planes k-1, k, k+1 and the output offset of plane
  // k-1, advanced with k.
  int ia = (kb + 2) % 3, ib = kb % 3, ic = (kb + 1) % 3;
  size_t g = (size_t)(kb - 1) * S + (size_t)gy * P + gx;
  // Unrolled by the intermediate ring's period (3): the slot indices and the
  // shift of the carried values resolve to fixed registers in each copy.
#pragma unroll 3
  for (int k = kb; k <= ke && !failed; ++k, g += S) {
    wait_plane(k + 2);
    failed = __syncthreads_or(failed);
    if (failed) break;
    issue(k + 4);
    // Both steps in one straight line, so that the second fills the first's
    // waits; a step that this iteration does not have (the first plane's second,
    // the last one's first) is computed from whatever is there and dropped.
    W wn;
    f2 l1p, c1p, c;
    const float *vk = sm.v1[ia];
    const f2 vp = ld2(&sm.ring[(k + 2) & (R - 1)].v[o]);
    const f2 t = kahan(wb, wza, l1b, vk[o1 - 1], vk[o1 + 2], ld2(&vk[o1 + V1X]), ld2(&vk[o1 - V1X]),
                       l1cc, l1a, c1b, c);
    level1(k + 1, vm, v0, vp, wzm, wn, l1p, c1p);
    if (l1_ok) *reinterpret_cast<f2 *>(&sm.v1[ic][o1]) = l1p;
    vm = v0;
    v0 = vp;
    wzm = wn.z;
    if (k > kb) {
      const unsigned cb = bf16(c);
      if (out0 && out1) {
        *reinterpret_cast<f2 *>(&vn[g]) = t;
        *reinterpret_cast<unsigned *>(&cn[g]) = cb;
      } else if (out0) {
        vn[g] = lo(t);
        cn[g] = (uint16_t)cb;
      } else if (out1) {
        vn[g + 1] = hi(t);
        cn[g + 1] = (uint16_t)(cb >> 16);
      }
    }
    l1a = l1b;
    l1b = l1cc;
    l1cc = l1p;
    c1b = c1cc;
    c1cc = c1p;
    wza = wb.z;
    wb = wcc;
    wcc = wn;
    const int t3 = ia;
    ia = ib;
    ib = ic;
    ic = t3;
  }
  if (failed) {
    if (tid == 0) atomicExch(err, 1);
    if (tid == 0) drain();
  }
}

__global__ void __launch_bounds__(NT, 2)
    k_fp32c_tb2(const __grid_constant__ Maps in, float *__restrict__ vn,
                uint16_t *__restrict__ cn, int nx, int ny, int nz, int P, size_t S, int kchunk,
                int *__restrict__ err, unsigned wait_limit) {
  const int kb = 1 + blockIdx.z * kchunk;
  const int ke = min(kb + kchunk, nz - 1);
  if (kb >= ke) return;
  tb2_tile(ParamMaps{in}, vn, cn, 1 + OX * blockIdx.x, 1 + OY * blockIdx.y, nx, ny, nz, P, S, kb,
           ke, err, wait_limit);
}

// The batch table's two-step FP32C tiles: one block per tile, hardware
// scheduled.  Grid g's maps are in device memory, seven per grid: v and carry
// of buffers 0 and 1, then wx, wy, wz; each launch reads buffer cur ^ flip.
__global__ void __launch_bounds__(NT, 2)
    k_batch_fp32c_tb2(const BatchGrid *__restrict__ grids, const BatchTile *__restrict__ tiles,
                      int flip) {
  const BatchTile tl = tiles[blockIdx.x];
  const BatchGrid &g = grids[tl.grid];
  const int src = g.cur ^ flip, dst = src ^ 1;
  const CUtensorMap *tm = static_cast<const CUtensorMap *>(g.tmaps);
  if (threadIdx.x == 0)  // the thread that issues the loads
    for (int m = 0; m < 7; ++m) tma::acquire_map(tm + m);
  __syncthreads();
  tb2_tile(TableMaps{tm, src}, (float *)g.f[dst], g.cr[dst], 1 + OX * tl.tx, 1 + OY * tl.ty, g.nx,
           g.ny, g.nz, g.P, g.S, tl.k0, tl.k1, g.err, kTableWaitLimit);
}

bool encode(CUtensorMap *m, const void *base, bool bf16, const heat_geom &g) {
  return tma::encode_field(m, base,
                           bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                           bf16 ? 2 : 4, g, bf16 ? BXC : BXF, BY);
}

constexpr size_t kSmem = sizeof(Smem) + 128;

// The kernels' shared memory allowed, once per process.
bool ready() {
  static const bool ok =
      cudaFuncSetAttribute(k_fp32c_tb2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) ==
          cudaSuccess &&
      cudaFuncSetAttribute(k_batch_fp32c_tb2, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kSmem) == cudaSuccess;
  return ok;
}

}  // namespace

int fp32c_tile_rows() { return OY; }

// A chunk's start costs about 4 planes' time: two planes of step t+1, their loads
// and the halo planes.
int fp32c_tb2_chunk(const heat_geom &g) {
  const long tiles = (long)((g.nx - 2 + OX - 1) / OX) * ((g.ny - 2 + OY - 1) / OY);
  static const long resident = ready() ? resident_blocks((const void *)k_fp32c_tb2, NT, kSmem) : 0;
  return balanced_chunk(tiles, g.nz - 2, resident, 4, 0.95, 128);
}

cudaError_t launch_batch_fp32c_tb2(const BatchGrid *grids, const BatchTile *tiles, int ntiles,
                                   int flip, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  if (!ready()) return cudaErrorInvalidConfiguration;
  k_batch_fp32c_tb2<<<ntiles, NT, kSmem, st>>>(grids, tiles, flip);
  return cudaGetLastError();
}

// False where the row and plane strides are not multiples of 16 bytes, which TMA
// wants (pitch a multiple of 8 points), or the encoder is missing.
bool encode_fp32c_maps(CUtensorMap *m, float *const v[2], uint16_t *const cr[2],
                       float *const w[3], const heat_geom &g) {
  return g.pitch % 8 == 0 && encode(&m[0], v[0], false, g) && encode(&m[1], v[1], false, g) &&
         encode(&m[2], cr[0], true, g) && encode(&m[3], cr[1], true, g) &&
         encode(&m[4], w[0], false, g) && encode(&m[5], w[1], false, g) &&
         encode(&m[6], w[2], false, g);
}

cudaError_t launch_fp32c_tb2(const heat_ctx *c, int cur, cudaStream_t st, unsigned wait_limit) {
  if (wait_limit > tma::kWaitLimit) wait_limit = tma::kWaitLimit;
  const heat_geom &g = c->g;
  if (!ready()) return cudaErrorInvalidConfiguration;
  const int kchunk = c->kchunk;
  dim3 grid((g.nx - 2 + OX - 1) / OX, (g.ny - 2 + OY - 1) / OY, (g.nz - 2 + kchunk - 1) / kchunk);
  return launch_chained(k_fp32c_tb2, grid, NT, kSmem, st,
                        Maps{c->maps[cur], c->maps[2 + cur], c->maps[4], c->maps[5], c->maps[6]},
                        c->v[cur ^ 1], c->carry[cur ^ 1], g.nx, g.ny, g.nz, g.pitch, g.plane,
                        kchunk, c->err, wait_limit);
}

}  // namespace heat
