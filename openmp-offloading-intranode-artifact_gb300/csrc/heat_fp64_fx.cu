// Default FP64 form: every point on the integer pipes, in fixed point at a
// scale shared by a 2 x 2 patch of columns.
//
// GB300 retires 2 FP64 operations per clock and SM, and 64 to 128 integer
// ones.  The update
//
//   u_new = uC + rhs + sum_f w_f (u_f - uC),   w_f = factor (kappa_a + kappa_b)
//
// (the reference's expression, OpenMP_Single_Source/heat3D_variable_coeff.c:
// 174-181, regrouped) costs 7 FP64 operations, which caps a kernel on the FP64
// pipe at 85 GLUP/s.  Here it is evaluated exactly but for the last bits of its
// products in 64-bit integers and rounded once:
//
//   * A thread owns a 2 x 2 patch of columns (rows j0 + 2m, j0 + 2m + 1, even
//     column i and i + 1) and walks planes.  At plane k its stencil region is
//     the patch at planes k - 1, k, k + 1 and the patch's eight in-plane
//     neighbours.  The largest exponent in the region (one more if any value
//     is negative, rounded up to an even number) gives the scale E: a value
//     becomes the integer A = value * 2^(1083 - E), |A| < 2^61.
//   * If no nonzero value of the patch itself (three planes) lies more than
//     kSlack = 8 binary orders below E, those A are exact, and are carried along
//     z.  Other values are cut to whole units, an error of one unit times the
//     weight.  A result below 2^53 units, where a unit is more than 1/2 ulp, is
//     formed anew on its own (2^51 where the region has both signs).
//   * Weights come from the per-point K = factor * kappa, kept as two limbs
//     K = k1 2^-32 + k0 2^-63 with |k0| <= 2^30: a face weight is the two limb
//     sums, no carry, and its low limb is a signed 32-bit number.
//   * Each face adds D w (D = A_f - A_C, limbs d1 signed, d0 unsigned) as three
//     32 x 32 -> 64 multiply-adds into exact accumulators: H += d1 w1,
//     X += round(D 2^-32) w0 (units of 2^-31), Y += d0 w1 (2^-32).  What that drops of
//     D w0 is at most half a unit and of either sign.  (With d1 for the rounded D it is
//     up to a whole unit, of one sign where the conductivity is constant: 300 steps at
//     the worst such value drifted by 1.0e-15, now 2e-19; 512^3 3 % faster.)
//     H + round(X, to two units) + round(Y) is then rounded to nearest even by one
//     int64 -> FP64 conversion (one operation of the FP64 pipe), and the scale goes into
//     its exponent field.
//
// The error of a step is that rounding (1/2 ulp of the result, at least one unit) and, in
// units: up to 6 x 1/2 for the six products, 1 and 1/2 for the sums, 6 x 1/4 for the
// weights, cut to 2^-63, and 1 for values cut to whole units: 7 at the very most, below
// one as a root mean square, against results of 2^53 units and more.  A sum of seven FP64
// multiply-adds has seven roundings, and rounded weights besides.  Largest relative error
// of a step (40^3, against 113 bits): random conductivity and field 1.1e-16 (5.2e-16 for
// the launch before the fixed point), a steep field 2.4e-16 (5.4e-16); after 30 steps
// 6.7e-16 (2.1e-15) and 5.6e-16 (2.5e-15).  A constant region stays exactly constant
// (every D is 0).
//
// Points formed on their own (results too small for their patch's units, patches without
// a scale: exponents near either end, infinities, NaNs) are aligned to the largest
// exponent of their own seven values.  Which way a point goes, and E, depend only on the
// field's values in the patch's region, never on tiles or z-chunks, so a grid's results
// are the same bits in any launch.  They are formed after the walk, from a list of
// patches or, where those are more than half of some planes, in a second walk.
//
// The integers carried along z move to a new scale by shifting, which is exact
// where both scales hold the patch exactly; elsewhere they are taken from the
// values again.  (Patches are small so that steep fields fit: of a Gaussian of
// width 0.05 on 512^3, whose tails fall by up to one binary order per point, no
// patch is outside the slack; of 16 x 8-point patches 40 % would be.)
//
// Staging: a block is 32 x 16 columns (128 threads, 16 x 8 patches).  Planes of
// u and K (and the source term) land by TMA in a ring 3 deep, boxes 36 x 18
// from column i0 - 2 (16-byte aligned), each slot completing on its own
// mbarrier; one block barrier per plane frees the oldest slot, whose next plane
// thread 0 then requests.
//
// Bound: the integer pipes and the latency between them.  At 512^3: 163 GLUP/s
// (0.814 ms a step; 133.5 for rows split between 7 FP64 operations and a per-point
// alignment in integers, the launch before the fixed point), with the reference's
// source term 153 (115.7); 192^3 with a narrow Gaussian 128.  155 instructions a point,
// with all the launch's share (300 for an integer row of that launch); at 320^3 the ALU
// pipe is 63 % busy, FMA 28 % (18 wide multiply-adds a point, each two of the others),
// FP64 45 %, issue 61 %, DRAM 24.7 bytes a point.
// Fields that the plain loop does not hold are slower (256^3, us a step, against the
// row-split launch's 137 to 198 for the same field): smooth 105, one sign throughout
// 120 to 125, zeros 80, random signs 139 at first and 170 once smooth (137), a
// front of 40 binary orders in zeros 117 at first and up to 250 while it spreads (190).
// Measured and not kept, each against the loop of its time (512^3, GLUP/s): the
// neighbours of one row converted by the FP64 pipe as the patch's own are, 169 for 173
// (157 for 167 of both); no value converted by it 164 for 167; five blocks per SM at 96
// registers 162 for 167; 32 x 32 tiles 156, 64 x 8 166, the plane loop unrolled by 2 162
// for the same 167.
//
// Every mbarrier wait is bounded: a wait that runs out stops the block at the
// next barrier (the flag is OR-reduced), thread 0 waits (bounded) for its loads
// in flight, *err is set and the host reports HEAT_ETIMEOUT.

#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "heat_batch_internal.h"
#include "heat_internal.h"
#include "heat_tma.cuh"

namespace heat {
namespace {

typedef unsigned long long u64;
typedef long long i64;

constexpr int TX = 32, TY = 16;          // columns of a tile
constexpr int NTX = TX / 2, NTY = TY / 2;
constexpr int NT = NTX * NTY;            // threads, one per 2 x 2 patch
constexpr int BX = TX + 4, BY = TY + 2;  // box: columns i0 - 2 .. i0 + 33, rows j0 - 1 .. j0 + 16
// Ring depth: planes k, k + 1 and one in flight (with a fourth slot 512^3 took
// 0.1 % longer, 256^3 0.7 %).
constexpr int kRing = 3;
constexpr int kMaxPlanes = 32;  // of a chunk: a bit each in `again`
constexpr int kMinB = 4;   // blocks per SM: 128 registers a thread, no spills

constexpr unsigned kExp = 1u << 20;      // one binary order in the high word of a double
constexpr unsigned kExpMask = 0x7ff00000u;
constexpr unsigned kSlack = 8 * kExp;
// A patch with a nonzero value this far below E (binary orders, in place) is left to be
// formed point by point: nearly all of its results would be too small.  (256^3, us a
// step: a hot cube in zeros, steps 20 to 220, 275 without, 245 at 13 orders, 252 at 16,
// 267 at 24; random signs 169, 171, 169, 168.)
constexpr unsigned kSteep = 14 * kExp;
constexpr unsigned kUnheld = 1;  // of a patch's scale: does not hold its plane before exactly
constexpr int kLeast = 1 << (53 - 32);          // high word of 2^53
constexpr int kLeastCrossing = 1 << (51 - 32);  // of 2^51
constexpr unsigned kLowE = 128 * kExp, kMidE = 1083 * kExp, kHighE = 2030 * kExp;

// Element count of `rows` box rows padded to 128 bytes: each array of a slot
// starts on a 128-byte boundary, as TMA shared-memory destinations must.
constexpr int pad128(int elems) { return (elems * 8 + 127) / 128 * 128 / 8; }
constexpr int kPad = pad128(BX * BY), kRPad = pad128(TX * TY);

template <bool RHS>
struct __align__(128) Slot {
  u64 u[kPad];
  u64 k[kPad];
};
template <>
struct __align__(128) Slot<true> {
  u64 u[kPad];
  u64 k[kPad];
  u64 r[kRPad];  // source term at the tile's own columns
};
template <bool RHS>
constexpr unsigned kSlotBytes = (2u * BX * BY + (RHS ? TX * TY : 0)) * 8u;
static_assert(sizeof(Slot<false>) % 128 == 0 && sizeof(Slot<true>) % 128 == 0 &&
                  (kPad * 8) % 128 == 0,
              "ring slots and their arrays start on 128-byte boundaries");

template <bool RHS>
struct Smem {
  Slot<RHS> ring[kRing];
  // Each thread's patch at the plane below where its registers do not hold it;
  // after the walk, the list of patches to form again.
  ulonglong2 below[2][NT];
  int count;        // of marked patches
  unsigned planes;  // that have some, a bit each
  u64 bar[kRing];
};

// Where a tile finds its tensor maps: kernel parameters for a single grid,
// device memory for a batch (u of buffers 0 and 1, K, source term).
struct Maps {
  CUtensorMap u, k, r;
};
struct ParamMaps {
  static constexpr bool kInMemory = false;
  static constexpr unsigned kLimit = kWaitLimit;
  const Maps &m;
  __device__ __forceinline__ const CUtensorMap *u() const { return &m.u; }
  __device__ __forceinline__ const CUtensorMap *k() const { return &m.k; }
  __device__ __forceinline__ const CUtensorMap *r() const { return &m.r; }
};
struct TableMaps {
  static constexpr bool kInMemory = true;
  static constexpr unsigned kLimit = kTableWaitLimit;
  const CUtensorMap *tm;
  int src;
  __device__ __forceinline__ const CUtensorMap *u() const { return &tm[src]; }
  __device__ __forceinline__ const CUtensorMap *k() const { return &tm[2]; }
  __device__ __forceinline__ const CUtensorMap *r() const { return &tm[3]; }
};

// Sizes and signs of a set of values, from their high words, an instruction or two
// each (masking the exponents first cost 1 % more in all).  Zeros do not count
// in mn (it wraps to the top); subnormals count as too small to be held, and
// beside a normal number are below 2^-60 units and read as 0.  fx_tile tells a
// region of zeros from one of subnormals.
struct Range {
  unsigned neg = 0;  // largest size of a negative value, its sign bit set
  int pos = 0;       // largest size of another one
  unsigned mn = ~0u; // smallest nonzero size, twice, less 2
  __device__ __forceinline__ void bound(u64 v) {
    const unsigned hi = (unsigned)(v >> 32);
    neg = max(neg, hi);
    pos = max(pos, (int)hi);
  }
  __device__ __forceinline__ void see(u64 v) {
    bound(v);
    mn = min(mn, (unsigned)(v >> 32) * 2u - 2u);
  }
  __device__ __forceinline__ void see(const Range &o) {
    neg = max(neg, o.neg);
    pos = max(pos, o.pos);
    mn = min(mn, o.mn);
  }
  __device__ __forceinline__ bool negative() const { return (int)neg < 0; }
  __device__ __forceinline__ bool crossing() const { return (int)neg < 0 && pos >= (int)kExp; }
  __device__ __forceinline__ unsigned size() const {
    return negative() ? max((unsigned)pos, neg & 0x7fffffffu) : (unsigned)pos;
  }
  // Scale (exponent field) of the region.
  __device__ __forceinline__ unsigned scale() const {
    const unsigned up = negative() ? 2 * kExp : kExp;
    return max((size() + up) & ~(2 * kExp - 1), kLowE);
  }
  __device__ __forceinline__ bool zero() const { return size() < kExp; }
  __device__ __forceinline__ bool steep(unsigned E) const { return mn < 2 * (E - kSteep) - 2; }
  // Whether the scale holds every value seen exactly.
  __device__ __forceinline__ bool held(unsigned E) const {
    return mn >= 2 * (E - kSlack) - 2 && E <= kHighE && !zero();
  }
};

__device__ __forceinline__ u64 shr(u64 a, unsigned n) {  // 0 for n >= 64
  u64 r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(n));
  return r;
}
__device__ __forceinline__ u64 sar(u64 a, unsigned n) {
  u64 r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(n));
  return r;
}
__device__ __forceinline__ u64 shl(u64 a, unsigned n) {
  u64 r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(n));
  return r;
}

// |v| in units of 2^(E - 1083): the significand left-aligned, its leading bit
// or-ed in, shifted right by 3 + E - e (over 63, so to 0, where the exponent
// field is 0).  The bits below the exponent do not matter to that difference once
// it is rounded up, so only a sign is masked.
template <bool SIGN>
__device__ __forceinline__ u64 magnitude(u64 v, unsigned E) {
  const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
  const unsigned h = __funnelshift_l(lo, hi, 11) | 0x80000000u;
  return shr(((u64)h << 32) | (lo << 11),
             (E + (4 * kExp - 1) - (SIGN ? hi & 0x7fffffffu : hi)) >> 20);
}
// The same of any value, subnormal ones exactly too.
__device__ __forceinline__ u64 magnitude_low(u64 v, unsigned E) {
  const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v, e = hi >> 20 & 0x7ff;
  const unsigned h = (__funnelshift_l(lo, hi, 11) & 0x7fffffffu) | (e ? 0x80000000u : 0u);
  return shr(((u64)h << 32) | (lo << 11), (E >> 20) + 3 - max(e, 1u));
}
// A value, with its sign, for E <= kMidE, by the FP64 pipe: the scale goes into the
// exponent field (0 stays below 1/2 unit) and the conversion does the rest.
__device__ __forceinline__ u64 convert(u64 v, unsigned E) {
  return (u64)__double2ll_rn(
      __hiloint2double((int)((unsigned)(v >> 32) + (kMidE - E)), (int)(unsigned)v));
}
__device__ __forceinline__ u64 with_sign(u64 a, u64 v) {
  const u64 s = (u64)((i64)v >> 63);
  return (a ^ s) - s;
}

// A value of point q of a patch, as the patch form rounds it where the scale does not
// hold it.
__device__ __forceinline__ u64 carried(u64 v, int q, unsigned E) {
  return q == 3 || E > kMidE ? with_sign(magnitude<true>(v, E), v) : convert(v, E);
}

// r units of 2^(E - 1083).
__device__ __forceinline__ double scaled(double r, unsigned E) {
  const unsigned hi = (unsigned)__double2hiint(r);  // 0 only for 0
  return __hiloint2double((int)(hi ? hi + (E - kMidE) : 0u), __double2loint(r));
}

template <bool B>
struct Bool {
  static constexpr bool value = B;
};

// Kinds of patch code: for values that are not negative, for any sign, and for scales
// above kMidE.  The first two round every value alike, so a patch of the first kind has
// the same bits in either.
constexpr int kPlain = 0, kSigned = 1, kAnyScale = 2;
template <int K>
struct Kind {
  static constexpr int value = K;
};

struct Acc {
  u64 H, X, Y;
  __device__ __forceinline__ explicit Acc(u64 centre) : H(centre), X(1ull << 31), Y(1ull << 31) {}
  // += D * w
  __device__ __forceinline__ void face(u64 D, unsigned w0, unsigned w1) {
    const unsigned d0 = (unsigned)D, d1 = (unsigned)(D >> 32);
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(H) : "r"(d1), "r"(w1));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(X) : "r"(d1 + (d0 >> 31)), "r"(w0));
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(Y) : "r"(d0), "r"(w1));
  }
  __device__ __forceinline__ void face(u64 D, u64 ka, u64 kb) {
    face(D, (unsigned)ka + (unsigned)kb, (unsigned)(ka >> 32) + (unsigned)(kb >> 32));
  }
  // The sum in units, to the nearest FP64 value.
  __device__ __forceinline__ double rounded() {
    asm("mad.wide.s32 %0, %1, 2, %0;" : "+l"(H) : "r"((unsigned)(X >> 32)));
    H += Y >> 32;
    return __ll2double_rn((i64)H);
  }
  // += v to the nearest unit
  __device__ __forceinline__ void add(u64 v, unsigned E) {
    const u64 h = magnitude<true>(v, E - kExp);  // in half units
    H += with_sign((h >> 1) + (h & 1), v);
  }
};

// A point's values and weights (f and k: above, below, west, east, south, north) and
// source term.
struct Stencil {
  u64 c, f[6], kc, k[6], vr;
};
// A point in FP64 operations.
template <bool RHS>
__device__ __forceinline__ double fp64_point(const Stencil &s) {
  const double uc = __longlong_as_double((i64)s.c);
  double acc = RHS ? uc + __longlong_as_double((i64)s.vr) : uc;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const int w0 = (int)((unsigned)s.kc + (unsigned)s.k[q]);
    const i64 w1 = (unsigned)(s.kc >> 32) + (unsigned)(s.k[q] >> 32);
    acc = fma((double)(w1 * (1ll << 31) + w0) * 0x1p-63, __longlong_as_double((i64)s.f[q]) - uc, acc);
  }
  return acc;
}
template <bool RHS>
__device__ __forceinline__ Range range(const Stencil &s) {
  Range r;
  r.bound(s.c);
#pragma unroll
  for (int q = 0; q < 6; ++q) r.bound(s.f[q]);
  if constexpr (RHS) r.bound(s.vr);
  return r;
}
__device__ __forceinline__ unsigned own_scale(const Range &r) {
  return (r.size() & kExpMask) + (r.negative() ? kExp : 0u);
}
// A point at scale E, a whole exponent.  LOW: for scales below kLowE too, where values
// and the result may be subnormal.
template <bool RHS, bool SIGN, bool LOW>
__device__ __forceinline__ double at_scale(const Stencil &s, unsigned E) {
  auto load = [&](u64 v) {
    const u64 m = LOW ? magnitude_low(v, E) : magnitude<SIGN>(v, E);
    return SIGN ? with_sign(m, v) : m;
  };
  const u64 A = load(s.c);
  Acc a(A);
#pragma unroll
  for (int q = 0; q < 6; ++q) a.face(load(s.f[q]) - A, s.kc, s.k[q]);
  if constexpr (RHS) {
    if (LOW) {
      const u64 h = magnitude_low(s.vr, E - kExp);
      a.H += with_sign((h >> 1) + (h & 1), s.vr);
    } else {
      a.add(s.vr, E);
    }
  }
  const bool up = LOW && E < kLowE;
  const double r = scaled(a.rounded(), up ? E + 200 * kExp : E);
  return up ? r * 0x1p-200 : r;
}

// One point with values of 2^1007 and more, by way of a power of two; infinities and
// NaNs in FP64 operations.
template <bool RHS>
__device__ __forceinline__ double high_point(Stencil &s) {
  if (range<RHS>(s).size() >= kExpMask) return fp64_point<RHS>(s);
  auto times = [](u64 &v) { v = (u64)__double_as_longlong(__longlong_as_double((i64)v) * 0x1p-200); };
  times(s.c);
#pragma unroll
  for (int q = 0; q < 6; ++q) times(s.f[q]);
  if constexpr (RHS) times(s.vr);
  return at_scale<RHS, true, false>(s, own_scale(range<RHS>(s))) * 0x1p200;
}

// The conductivities themselves, for results that live on small weights.
struct Kappa {
  const double *k;  // the grid's
  double factor;
  int P;
  size_t S;
};
// A point, at offset g, of values that are all of one sign (so that nothing cancels) and
// weights below 2^-20, of which K has 43 bits and fewer: in FP64 operations of the
// conductivities.  (Insulators of 1e-9 among conductors, cold at first: largest relative
// error after 10 steps 6.5e-9 without, 1.5e-9 so; 5.5e-9 for the launch before the fixed
// point.  A hot cube in zeros at 256^3 255 us a step without, 275 so.)
template <bool RHS>
__device__ __forceinline__ double weak_point(const Stencil &s, const Kappa &kap, size_t g) {
  const double *k = kap.k + g;
  const size_t S = kap.S;
  const int P = kap.P;
  const double kf[6] = {__ldcg(k + S), __ldcg(k - S), __ldcg(k - 1),
                        __ldcg(k + 1), __ldcg(k - P), __ldcg(k + P)};
  const double kc = __ldcg(k), uc = __longlong_as_double((i64)s.c);
  double sum = 0.0;
#pragma unroll
  for (int q = 0; q < 6; ++q) sum = fma(kc + kf[q], __longlong_as_double((i64)s.f[q]) - uc, sum);
  return fma(kap.factor, sum, RHS ? uc + __longlong_as_double((i64)s.vr) : uc);
}
// N points, at offsets g, from their values and weights, in one straight line: the same
// arithmetic at each point's own scale, the largest exponent of its seven values (and the
// source term), every value cut to that scale's units.
template <bool RHS, int N>
__device__ __forceinline__ void points(Stencil (&s)[N], const Kappa &kap, const size_t (&g)[N],
                                       double (&out)[N]) {
  unsigned E[N];
  bool neg = false, low = false, high = false, one_sign[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const Range r = range<RHS>(s[n]);
    E[n] = max(own_scale(r), 2 * kExp);
    one_sign[n] = !r.crossing() && E[n] <= kHighE;
    neg |= r.negative();
    low |= E[n] < kLowE;
    high |= E[n] > kHighE;
  }
  auto all = [&](auto sign, auto subnormal) {
#pragma unroll
    for (int n = 0; n < N; ++n) out[n] = at_scale<RHS, sign.value, subnormal.value>(s[n], E[n]);
  };
  if (low)
    all(Bool<true>{}, Bool<true>{});
  else if (neg)
    all(Bool<true>{}, Bool<false>{});
  else
    all(Bool<false>{}, Bool<false>{});
  if (high)
#pragma unroll
    for (int n = 0; n < N; ++n)
      if (E[n] > kHighE) out[n] = high_point<RHS>(s[n]);
  // A result of fewer than 2^46 units by such weights alone.
#pragma unroll
  for (int n = 0; n < N; ++n)
    if (((unsigned)__double2hiint(out[n]) & 0x7fffffffu) + 14 * kExp < E[n] && one_sign[n]) {
      unsigned top = 0;  // the largest weight's high limb, units of 2^-32
#pragma unroll
      for (int q = 0; q < 6; ++q) top = max(top, (unsigned)(s[n].k[q] >> 32));
      if (top + (unsigned)(s[n].kc >> 32) < 1u << 12) out[n] = weak_point<RHS>(s[n], kap, g[n]);
    }
}

// The points of the marked patches (bit p of a thread's `again`: plane kb + p),
// each on its own, four lanes to a patch: the whole block lists them in `list`
// (16 planes of it at a time) and takes 32 at a time.  104 x 107 x 63 with a
// narrow Gaussian, where 9 % of the patches are marked at first: 13.0 us a step
// (48 steps); 16.2 with each thread going over its own.
template <bool RHS>
__device__ __noinline__ void form_alone(unsigned again, unsigned short *list, int *count,
                                        double *un, const u64 *u, const u64 *K, const u64 *rhs,
                                        Kappa kap, int tx, int ty, int kb, int nx, int ny, int P,
                                        size_t S) {
  const int me = threadIdx.x;
  for (int first = 0; first < kMaxPlanes; first += 16) {
    __syncthreads();
    if (me == 0) *count = 0;
    __syncthreads();
    unsigned m = again >> first & 0xffffu;
    if (m)
      for (int at = atomicAdd(count, __popc(m)); m; m &= m - 1)
        list[at++] = (unsigned short)((first + __ffs(m) - 1) * NT + me);
    __syncthreads();
    const int n = *count;
#pragma unroll 1
    for (int e = me / 4; e < n; e += NT / 4) {
      const int t = list[e] % NT, k = kb + list[e] / NT;
      const int i = tx * TX + 2 * (t % NTX) + (me & 1);
      const int j = 1 + ty * TY + 2 * (t / NTX) + (me >> 1 & 1);
      if (i < 1 || i >= nx - 1 || j >= ny - 1) continue;
      const size_t g[1] = {(size_t)k * S + (size_t)j * P + i};
      const u64 *v = u + g[0], *kv = K + g[0];
      Stencil st[1] = {{__ldcg(v),
                        {__ldcg(v + S), __ldcg(v - S), __ldcg(v - 1), __ldcg(v + 1), __ldcg(v - P),
                         __ldcg(v + P)},
                        __ldcg(kv),
                        {__ldcg(kv + S), __ldcg(kv - S), __ldcg(kv - 1), __ldcg(kv + 1),
                         __ldcg(kv - P), __ldcg(kv + P)},
                        RHS ? __ldcg(rhs + g[0]) : 0}};
      double out[1];
      points<RHS>(st, kap, g, out);
      un[g[0]] = out[0];
    }
  }
}

__device__ __forceinline__ ulonglong2 ld2(const u64 *p) {
  return *reinterpret_cast<const ulonglong2 *>(p);
}

// Keeps the compiler from holding values read before this point in registers.
__device__ __forceinline__ void reload() { asm volatile("" ::: "memory"); }

// The marked patches in a second walk, over the planes from kb + first to kb + last: the
// same points from the ring, whose n loads of the first walk give the parities.  Returns
// true if a wait ran out.  Bound: integer instructions, 220 a point.  256^3 where every
// patch has values 2^40 apart: 274 us a step, 584 from the list; a hot cube in zeros,
// steps 20 to 220, 249 for 390.  Forming such patches inside the first walk costs that
// its schedule (512^3: 804 to 850 us a step for 770).
template <bool RHS, class M>
__device__ __noinline__ bool form_walk(const M maps, Smem<RHS> &sm, unsigned again, int n,
                                       double *un, Kappa kap, int tx, int ty, int nx, int ny, int P,
                                       size_t S, int kb, int first, int last, unsigned wait_limit) {
  const int t = threadIdx.x, lx = t % NTX, ly = t / NTX;
  const int i = tx * TX + 2 * lx, j = 1 + ty * TY + 2 * ly, o = (2 * ly + 1) * BX + 2 * lx + 2;
  const bool x0 = i >= 1 && i < nx - 1, x1 = i + 1 < nx - 1;
  const bool y0 = j < ny - 1, y1 = j + 1 < ny - 1;
  const int k0 = kb + first, ke = kb + last + 1, planes = ke - k0 + 2;
  auto issue = [&](int p) {  // plane k0 - 1 + p
    if (t != 0 || p >= planes) return;
    Slot<RHS> &sl = sm.ring[p % kRing];
    u64 *b = &sm.bar[p % kRing];
    tma::fence_proxy_async();
    tma::mbar_expect(b, kSlotBytes<RHS>);
    tma::load3(sl.u, maps.u(), tx * TX - 2, ty * TY, k0 - 1 + p, b);
    tma::load3(sl.k, maps.k(), tx * TX - 2, ty * TY, k0 - 1 + p, b);
    if constexpr (RHS) tma::load3(sl.r, maps.r(), tx * TX, ty * TY + 1, k0 - 1 + p, b);
  };
  auto wait = [&](int p, unsigned limit) {
    const int s = p % kRing;
    return tma::mbar_wait(&sm.bar[s], ((n - s + kRing - 1) / kRing + p / kRing) & 1u, limit);
  };
  for (int p = 0; p < kRing; ++p) issue(p);
  bool failed = !wait(0, wait_limit) || !wait(1, wait_limit);
  u64 lo[4], kl[4];  // the patch below and its weights
  auto below = [&](const Slot<RHS> &s) {
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const ulonglong2 v = ld2(&s.u[o + y * BX]), k = ld2(&s.k[o + y * BX]);
      lo[2 * y] = v.x, lo[2 * y + 1] = v.y, kl[2 * y] = k.x, kl[2 * y + 1] = k.y;
    }
  };
  below(sm.ring[0]);
  double *w = un + (size_t)k0 * S + (size_t)j * P + i;
  int p = 1;  // of plane k
  for (int k = k0; k < ke; ++k, ++p, w += S) {
    if (!failed) failed = !wait(p + 1, wait_limit);
    failed = __syncthreads_or(failed);
    if (failed) break;
    issue(p - 1 + kRing);
    const Slot<RHS> &sk = sm.ring[p % kRing], &sn = sm.ring[(p + 1) % kRing];
    if (again >> (k - kb) & 1u) {
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        if (!(y ? y1 : y0)) continue;
        Stencil st[2];
        double out[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int c = o + y * BX + x, q = 2 * y + x;
          st[x] = {sk.u[c],
                   {sn.u[c], lo[q], sk.u[c - 1], sk.u[c + 1], sk.u[c - BX], sk.u[c + BX]},
                   sk.k[c],
                   {sn.k[c], kl[q], sk.k[c - 1], sk.k[c + 1], sk.k[c - BX], sk.k[c + BX]},
                   0};
          if constexpr (RHS) st[x].vr = sk.r[(2 * ly + y) * TX + 2 * lx + x];
        }
        const size_t g = w - un + (y ? P : 0);
        points<RHS>(st, kap, {g, g + 1}, out);
        if (x0) w[y ? P : 0] = out[0];
        if (x1) w[(y ? P : 0) + 1] = out[1];
      }
    }
    below(sk);
  }
  // Planes p - 1 and on were requested up to p + kRing - 2.
  if (failed && t == 0)
    for (int q = p - 1; q <= min(p + kRing - 2, planes - 1); ++q) wait(q, M::kLimit);
  return failed;
}

// One step over the (32 x 16)-column tile (tx, ty), planes [kb, ke), of the
// field u into un; at most kMaxPlanes planes.  Returns true if a wait ran out, here or
// in a launch before (*err).
template <bool RHS, class M>
__device__ __forceinline__ bool fx_tile(const M &maps, Smem<RHS> &sm, double *__restrict__ un,
                                        const u64 *__restrict__ u, const u64 *__restrict__ K,
                                        const u64 *__restrict__ rhs, const double *kappa,
                                        double factor, int tx, int ty, int nx, int ny, int P,
                                        size_t S, int kb, int ke, const int *err,
                                        unsigned wait_limit) {
  const int t = threadIdx.x, lx = t % NTX, ly = t / NTX;
  const int i = tx * TX + 2 * lx, j = 1 + ty * TY + 2 * ly;  // patch: i, i + 1; j, j + 1
  const int o = (2 * ly + 1) * BX + 2 * lx + 2;              // its first point in a box
  const bool x0 = i >= 1 && i < nx - 1, x1 = i + 1 < nx - 1;
  const bool y0 = j < ny - 1, y1 = j + 1 < ny - 1;
  const bool active = y0 && (x0 || x1);  // the patch holds a point to write

  if (t == 0) {
    for (int s = 0; s < kRing; ++s) tma::mbar_init(&sm.bar[s]);
    tma::mbar_init_fence();
  }
  chain();
  auto issue = [&](int p, int s) {
    if (t != 0 || p > ke) return;
    Slot<RHS> &sl = sm.ring[s];
    u64 *b = &sm.bar[s];
    tma::fence_proxy_async();
    tma::mbar_expect(b, kSlotBytes<RHS>);
    tma::load3(sl.u, maps.u(), tx * TX - 2, ty * TY, p, b);
    tma::load3(sl.k, maps.k(), tx * TX - 2, ty * TY, p, b);
    if constexpr (RHS) tma::load3(sl.r, maps.r(), tx * TX, ty * TY + 1, p, b);
  };
  // The flag is read before the first loads where a wrong map could be what set it, else
  // beside them by another warp, and looked at with the first plane (40 x 33 x 28: 4.63 us
  // a step, 4.82 with the wait for it behind the loads).
  bool stop = t == (M::kInMemory ? 0 : NT - 1) && tma::gave_up(err);
  if (M::kInMemory) {
    if (__syncthreads_or(stop)) return true;
    stop = false;
  }
  for (int s = 0; s < kRing; ++s) issue(kb - 1 + s, s);
  if (!M::kInMemory) __syncthreads();

  // Carried along z, points in the order (i, j), (i + 1, j), (i, j + 1),
  // (i + 1, j + 1): the patch at plane k (A1) and its difference to plane k - 1
  // (Dd) at scale E (0: none yet), the weight limbs of the face below and the
  // ranges.
  u64 Dd[4], A1[4];
  unsigned W0[4], W1[4];
  Range r0, r1;
  unsigned E = 0;
  bool failed = !tma::mbar_wait(&sm.bar[0], 0, wait_limit) ||
                !tma::mbar_wait(&sm.bar[1], 0, wait_limit);
  if (!failed) {
    u64 a[4], b[4], ka[4], Kc[4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      ulonglong2 v = ld2(&sm.ring[0].u[o + q * BX]);
      a[2 * q] = v.x, a[2 * q + 1] = v.y;
      v = ld2(&sm.ring[1].u[o + q * BX]);
      b[2 * q] = v.x, b[2 * q + 1] = v.y;
      v = ld2(&sm.ring[0].k[o + q * BX]);
      ka[2 * q] = v.x, ka[2 * q + 1] = v.y;
      v = ld2(&sm.ring[1].k[o + q * BX]);
      Kc[2 * q] = v.x, Kc[2 * q + 1] = v.y;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      r0.see(a[q]);
      r1.see(b[q]);
      W0[q] = (unsigned)ka[q] + (unsigned)Kc[q];
      W1[q] = (unsigned)(ka[q] >> 32) + (unsigned)(Kc[q] >> 32);
    }
    Range r = r0;
    r.see(r1);
    E = r.scale();  // at most the first plane's scale, so what that needs exact is exact
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      A1[q] = with_sign(magnitude<true>(b[q], E), b[q]);
      Dd[q] = with_sign(magnitude<true>(a[q], E), a[q]) - A1[q];
    }
    if (!r.held(E)) {
      E = kUnheld;
      sm.below[0][t] = make_ulonglong2(a[0], a[1]);
      sm.below[1][t] = make_ulonglong2(a[2], a[3]);
    }
  }

  failed |= stop;
  // Slots of planes k - 1 and k at the top of an iteration, and the parity of
  // the next plane's phase.
  int s0 = 0, s1 = 1;
  unsigned parity = 0;
  double *w = un + (size_t)kb * S + (size_t)j * P + i;  // the patch at plane k
  // Keeps points that are not written out of `least`.
  const int skip[4] = {x0 && y0 ? 0 : 0x7fffffff, x1 && y0 ? 0 : 0x7fffffff,
                       x0 && y1 ? 0 : 0x7fffffff, x1 && y1 ? 0 : 0x7fffffff};
  unsigned again = 0;  // bit p: the patch at plane kb + p is to be formed point by point
  int k = kb;
  for (; k < ke; ++k, w += S) {
    const int s2 = s1 == kRing - 1 ? 0 : s1 + 1;
    if (s2 == 0) parity ^= 1;
    if (!failed) failed = !tma::mbar_wait(&sm.bar[s2], parity, wait_limit);
    failed = __syncthreads_or(failed);
    if (failed) break;
    issue(k - 1 + kRing, s0);  // every thread is done with plane k - 1
    const Slot<RHS> &sk = sm.ring[s1], &sn = sm.ring[s2];

    s0 = s1;
    s1 = s2;
    if (!active) continue;
    Range r2, r = r0;
    {
      u64 up[4], h[8];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        ulonglong2 v = ld2(&sn.u[o + q * BX]);
        up[2 * q] = v.x, up[2 * q + 1] = v.y;
        h[q] = sk.u[o + q * BX - 1];
        h[2 + q] = sk.u[o + q * BX + 2];
        v = ld2(&sk.u[q ? o + 2 * BX : o - BX]);
        h[4 + 2 * q] = v.x, h[5 + 2 * q] = v.y;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) r2.see(up[q]);
      r.see(r1);
      r.see(r2);
#pragma unroll
      for (int q = 0; q < 8; ++q) r.bound(h[q]);
    }
    u64 rr[4];
    if constexpr (RHS) {
      // The source counts towards the largest exponent only: it is added to
      // the nearest unit.
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        rr[q] = sk.r[(2 * ly + (q >> 1)) * TX + 2 * lx + (q & 1)];
        r.bound(rr[q]);
      }
    }
    const unsigned En = r.scale();
    const bool held = r.held(En);
    // Results of fewer units than this are formed on their own.  Where the field changes
    // sign a small result is mostly the difference of large terms, to which rounded
    // FP64 operations add more than the fixed point does, and fewer are (random signs at
    // 256^3: 164 us a step at first and 200 later with 2^53, 135 and 168 so; 512^3
    // without signs 812, 820 so).
    const int enough = r.crossing() ? kLeastCrossing : kLeast;
    int least = 0;  // high word of the smallest result (its size), in units
    if (!r.zero() && En <= kHighE && !r.steep(En)) {
      if ((E & ~kUnheld) != En) {
        if (!(E & kUnheld) && held) {
          const int d = (int)(En - E) >> 20;
          const unsigned dn = (unsigned)max(d, 0), ups = (unsigned)max(-d, 0);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            Dd[q] = sar(shl(Dd[q], ups), dn);
            A1[q] = sar(shl(A1[q], ups), dn);
          }
        } else {  // from the values: those below are A1 + Dd units, or in shared memory
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            u64 a = (u64)__double_as_longlong(scaled(__ll2double_rn((i64)(A1[q] + Dd[q])), E));
            if (E & kUnheld) a = q & 1 ? sm.below[q >> 1][t].y : sm.below[q >> 1][t].x;
            const u64 b = sk.u[o + (q >> 1) * BX + (q & 1)];
            A1[q] = carried(b, q, En);
            Dd[q] = carried(a, q, En) - A1[q];
          }
        }
      }
      E = En;
      // The values are read from shared memory again here, row by row, rather
      // than kept in registers from the range pass.
      u64 A2[4];
      least = 0x7fffffff;
      double out[4];
      auto patch = [&](auto kind) {
        // One straight line, no branch in it: with one between the points the
        // compiler forms them one after the other (512^3: 870 to 960 us a step for
        // 788).
        constexpr bool plain = kind.value == kPlain;
        auto load = [&](u64 v) {
          const u64 m = magnitude<!plain>(v, E);
          return plain ? m : with_sign(m, v);
        };
        reload();
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const int oy = o + y * BX, oo = y ? o + 2 * BX : o - BX;
          // of the row: the plane above (U), beside it (S), the other row of the
          // patch (I) and the one outside it (O)
          const ulonglong2 vU = ld2(&sn.u[oy]), vO = ld2(&sk.u[oo]);
          const ulonglong2 kC = ld2(&sk.k[oy]), kI = ld2(&sk.k[y ? o : o + BX]);
          const ulonglong2 kO = ld2(&sk.k[oo]), kU = ld2(&sn.k[oy]);
          const u64 vS[2] = {sk.u[oy - 1], sk.u[oy + 2]}, kS[2] = {sk.k[oy - 1], sk.k[oy + 2]};
          const u64 kc[2] = {kC.x, kC.y}, ki[2] = {kI.x, kI.y}, ko[2] = {kO.x, kO.y};
          const u64 ku[2] = {kU.x, kU.y}, vo[2] = {vO.x, vO.y};
          const int q0 = 2 * y;
          A2[q0] = kind.value != kAnyScale ? convert(vU.x, E) : load(vU.x);
          // (the fourth on the integer pipes: with the source term 823 us a step at 512^3,
          // 862 with all four converted, 819 with two; without 763, 766, 771)
          A2[q0 + 1] = kind.value != kAnyScale && y == 0 ? convert(vU.y, E) : load(vU.y);
          Acc a[2] = {Acc(A1[q0]), Acc(A1[q0 + 1])};
#pragma unroll
          for (int x = 0; x < 2; ++x) a[x].face(Dd[q0 + x], W0[q0 + x], W1[q0 + x]);
#pragma unroll
          for (int x = 0; x < 2; ++x) a[x].face(A1[q0 + (x ^ 1)] - A1[q0 + x], kc[x], kc[x ^ 1]);
#pragma unroll
          for (int x = 0; x < 2; ++x) a[x].face(A1[(q0 + x) ^ 2] - A1[q0 + x], kc[x], ki[x]);
#pragma unroll
          for (int x = 0; x < 2; ++x) a[x].face(load(vS[x]) - A1[q0 + x], kc[x], kS[x]);
#pragma unroll
          for (int x = 0; x < 2; ++x) a[x].face(load(vo[x]) - A1[q0 + x], kc[x], ko[x]);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int q = q0 + x;
            W0[q] = (unsigned)kc[x] + (unsigned)ku[x];
            W1[q] = (unsigned)(kc[x] >> 32) + (unsigned)(ku[x] >> 32);
            a[x].face(A2[q] - A1[q], W0[q], W1[q]);
            Dd[q] = A1[q] - A2[q];
            if constexpr (RHS) {
              if (kind.value != kAnyScale)
                a[x].H += convert(rr[q], E);
              else
                a[x].add(rr[q], E);
            }
          }
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int q = q0 + x;
            const double v = a[x].rounded();
            const int h = (int)(a[x].H >> 32);
            least = min(least, (plain ? h : h ^ (h >> 31)) | skip[q]);
            // (0 comes out wrong, but is below kLeast, and formed again.)
            out[q] = __hiloint2double(__double2hiint(v) + (int)(E - kMidE), __double2loint(v));
          }
        }
      };
      // One negative value and the lanes that are together take the code for any sign:
      // apart they cost both (random signs at 256^3, once smooth: 191 us a step without
      // the points formed again, 147 so).
      if (E > kMidE)
        patch(Kind<kAnyScale>{});
      else if (cooperative_groups::coalesced_threads().any(r.negative()))
        patch(Kind<kSigned>{});
      else
        patch(Kind<kPlain>{});
#pragma unroll
      for (int q = 0; q < 4; ++q) A1[q] = A2[q];
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        if (!(y ? y1 : y0)) continue;
        double *wy = w + (y ? P : 0);
        if (x0 && x1) {
          *reinterpret_cast<double2 *>(wy) = make_double2(out[2 * y], out[2 * y + 1]);
        } else {
          if (x0) wy[0] = out[2 * y];
          if (x1) wy[1] = out[2 * y + 1];
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int p = o + (q >> 1) * BX + (q & 1);
        const u64 Kc = sk.k[p], Ku = sn.k[p];
        W0[q] = (unsigned)Kc + (unsigned)Ku;
        W1[q] = (unsigned)(Kc >> 32) + (unsigned)(Ku >> 32);
      }
      // Zeros all around (of either sign; the patch below, not held, is in shared memory)
      // give zeros, without a mark: a body that is cold but for a spot is mostly this
      // (256^3 of zeros: 81 us a step, 540 with every point formed again).
      if ((E & kUnheld) && r.zero()) {
        u64 any = 0;
        auto with = [&](const ulonglong2 &v) { any |= v.x | v.y; };
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          with(sm.below[q][t]);
          with(ld2(&sk.u[o + q * BX]));
          with(ld2(&sn.u[o + q * BX]));
          with(ld2(&sk.u[q ? o + 2 * BX : o - BX]));
          any |= sk.u[o + q * BX - 1] | sk.u[o + q * BX + 2];
        }
        if constexpr (RHS) any |= rr[0] | rr[1] | rr[2] | rr[3];
        if (any << 1 == 0) {
          least = kLeast;
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            if (!(y ? y1 : y0)) continue;
            double *wy = w + (y ? P : 0);
            if (x0) wy[0] = 0.0;
            if (x1) wy[1] = 0.0;
          }
        }
      }
      E = 0;
    }
    if (!held) {
      E |= kUnheld;
      sm.below[0][t] = ld2(&sk.u[o]);
      sm.below[1][t] = ld2(&sk.u[o + BX]);
    }
    // No scale, values too far apart, or a result too small for its units (zeros in the
    // patch, small neighbours).
    if (least < enough) again |= 1u << (k - kb);
    r0 = r1;
    r1 = r2;
  }
  // Planes k - 1 and on were requested up to plane k + kRing - 2.
  if (failed && t == 0)
    for (int p = k - 1; p <= min(k + kRing - 2, ke); ++p)
      tma::mbar_wait(&sm.bar[(p - kb + 1) % kRing], (p - kb + 1) / kRing & 1u, M::kLimit);
  // Formed after the walk: inside it, inlined or called, it costs the loop its schedule
  // (512^3: 808 to 930 us a step for 788).  A plane of the second walk takes about as
  // long as half its patches from the list (104 x 107 x 63 with a narrow Gaussian 13.8 us
  // a step; 15.4 with the line at a quarter).
  if (!__syncthreads_or(again != 0 && !failed)) return failed;
  if (t == 0) sm.count = 0, sm.planes = 0;
  __syncthreads();
  const unsigned some = __reduce_or_sync(~0u, again), many = __reduce_add_sync(~0u, __popc(again));
  if (t % 32 == 0) {
    atomicAdd(&sm.count, (int)many);
    atomicOr(&sm.planes, some);
  }
  __syncthreads();
  const Kappa kap{kappa, factor, P, S};
  const int first = __ffs(sm.planes) - 1, last = 31 - __clz(sm.planes);
  if (2 * sm.count > NT * (last - first + 1))
    return form_walk<RHS>(maps, sm, again, ke - kb + 2, un, kap, tx, ty, nx, ny, P, S, kb, first, last,
                          wait_limit);
  form_alone<RHS>(again, reinterpret_cast<unsigned short *>(sm.below), &sm.count, un, u, K, rhs, kap,
                  tx, ty, kb, nx, ny, P, S);
  return failed;
}

template <bool RHS>
__device__ __forceinline__ Smem<RHS> &smem() {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  return *reinterpret_cast<Smem<RHS> *>(smem_raw);
}

template <bool RHS>
__global__ void __launch_bounds__(NT, kMinB)
    k_fx(const __grid_constant__ Maps maps, double *__restrict__ un, const u64 *__restrict__ u,
         const u64 *__restrict__ K, const u64 *__restrict__ rhs, const double *__restrict__ kappa,
         double factor, int nx, int ny, int nz, int P, size_t S, int k0, int kchunk, int *__restrict__ err, unsigned wait_limit) {
  const int kb = k0 + blockIdx.z * kchunk;
  const int ke = min(kb + kchunk, nz - 1);
  if (kb >= ke) return;  // whole block
  if (fx_tile<RHS>(ParamMaps{maps}, smem<RHS>(), un, u, K, rhs, kappa, factor, blockIdx.x, blockIdx.y, nx, ny, P,
                   S, kb, ke, err, wait_limit) &&
      threadIdx.x == 0)
    atomicExch(err, 1);
}

// The batch table's tiles: one block per tile.  Grid g's maps are in device
// memory, four per grid; each launch reads buffer cur ^ flip.
template <bool RHS>
__global__ void __launch_bounds__(NT, kMinB)
    k_batch_fx(const BatchGrid *__restrict__ grids, const BatchTile *__restrict__ tiles, int flip) {
  const BatchTile tl = tiles[blockIdx.x];
  const BatchGrid &g = grids[tl.grid];
  const int src = g.cur ^ flip, dst = src ^ 1;
  const CUtensorMap *tm = static_cast<const CUtensorMap *>(g.tmaps);
  // By the thread that issues the loads, for each map: a fence orders its own
  // thread's accesses.
  if (threadIdx.x == 0)
    for (int m = 0; m < 4; ++m) tma::acquire_map(tm + m);
  __syncthreads();
  if (fx_tile<RHS>(TableMaps{tm, src}, smem<RHS>(), (double *)g.f[dst], (const u64 *)g.f[src], g.kq,
                   (const u64 *)g.rhs, (const double *)g.w[0], g.factor, tl.tx, tl.ty, g.nx, g.ny, g.P, g.S, tl.k0, tl.k1,
                   g.err, kTableWaitLimit) &&
      threadIdx.x == 0)
    atomicExch(g.err, 1);
}

template <bool RHS>
constexpr size_t smem_bytes() { return sizeof(Smem<RHS>) + 128; }

bool allow_smem(const void *kernel, size_t bytes) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) ==
      cudaSuccess)
    return true;
  cudaGetLastError();
  return false;
}

template <bool RHS>
bool usable() {
  static const bool ok = tma::encoder() && allow_smem((const void *)k_fx<RHS>, smem_bytes<RHS>()) &&
                         allow_smem((const void *)k_batch_fx<RHS>, smem_bytes<RHS>());
  return ok;
}

bool encode(CUtensorMap *m, const void *base, const heat_geom &g, unsigned x, unsigned y) {
  return tma::encode_field(m, base, CU_TENSOR_MAP_DATA_TYPE_UINT64, 8, g, x, y);
}

template <bool RHS>
long resident() {
  static const long n = resident_blocks((const void *)k_fx<RHS>, NT, smem_bytes<RHS>());
  return n;
}

template <bool RHS>
cudaError_t launch(const heat_ctx *c, int cur, cudaStream_t st, unsigned wait_limit) {
  const heat_geom &g = c->g;
  const int kc = c->kchunk;
  // A chunk has at most kMaxPlanes planes and a launch kMaxGridZ chunks: past 2 M
  // planes a step takes several launches.
  cudaError_t e = cudaSuccess;
  for (int k0 = 1, left = (g.nz - 2 + kc - 1) / kc; left > 0 && e == cudaSuccess;
       left -= kMaxGridZ, k0 += kMaxGridZ * kc)
    e = launch_chained(k_fx<RHS>, dim3(fx_tiles_x(g.nx), fx_tiles_y(g.ny), std::min(left, kMaxGridZ)),
                       NT, smem_bytes<RHS>(), st, Maps{c->maps[cur], c->maps[2], c->maps[3]},
                       c->u[cur ^ 1], (const u64 *)c->u[cur], c->kq, (const u64 *)c->rhs, c->kappa,
                       c->factor, g.nx, g.ny, g.nz, g.pitch, g.plane, k0, kc, c->err, wait_limit);
  return e;
}

}  // namespace

// Tiles start at column 0 (an even, 16-byte aligned column; it is a boundary
// column and not written) and row 1.
int fx_tiles_x(int nx) { return (nx - 1 + TX - 1) / TX; }
int fx_tiles_y(int ny) { return (ny - 2 + TY - 1) / TY; }

// Short tiles until a table holds 1.7 blocks for every resident one, as a small
// grid alone wants (64^3: 4.8 us a step at 1 plane, 6.7 at 2, 9.9 at 8); never
// more than kMaxPlanes.
int fx_fill_chunk(long tile_planes, bool rhs) {
  const long n = rhs ? resident<true>() : resident<false>();
  const long kc = n > 0 ? (3 * tile_planes + 5 * n - 1) / (5 * n) : 16;
  return kc < 1 ? 1 : kc < kMaxPlanes ? (int)kc : kMaxPlanes;
}

// A chunk's start, its first loads, costs about a plane's time; 384^3 runs 329 us
// a step at 20 planes, 355 at 191.
int fx_chunk(const heat_geom &g, bool rhs) {
  return balanced_chunk((long)fx_tiles_x(g.nx) * fx_tiles_y(g.ny),
                        std::min(g.nz - 2, kMaxGridZ * kMaxPlanes),
                        rhs ? resident<true>() : resident<false>(), 1, 0.53, kMaxPlanes);
}

bool fx_usable(bool rhs) { return rhs ? usable<true>() : usable<false>(); }

bool encode_fx_maps(CUtensorMap *m, double *const u[2], const unsigned long long *K,
                    const double *rhs, const heat_geom &g) {
  if (!rhs) std::memset(&m[3], 0, sizeof m[3]);
  return encode(&m[0], u[0], g, BX, BY) && encode(&m[1], u[1], g, BX, BY) &&
         encode(&m[2], K, g, BX, BY) && (!rhs || encode(&m[3], rhs, g, TX, TY));
}

cudaError_t launch_fx(const heat_ctx *c, int cur, cudaStream_t st, unsigned wait_limit) {
  if (!fx_usable(c->rhs != nullptr)) return cudaErrorInvalidConfiguration;
  if (wait_limit > kWaitLimit) wait_limit = kWaitLimit;
  return c->rhs ? launch<true>(c, cur, st, wait_limit) : launch<false>(c, cur, st, wait_limit);
}

cudaError_t launch_batch_fx(const BatchGrid *grids, const BatchTile *tiles, int ntiles, bool rhs,
                            int flip, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  if (!fx_usable(rhs)) return cudaErrorInvalidConfiguration;
  if (rhs)
    k_batch_fx<true><<<ntiles, NT, smem_bytes<true>(), st>>>(grids, tiles, flip);
  else
    k_batch_fx<false><<<ntiles, NT, smem_bytes<false>(), st>>>(grids, tiles, flip);
  return cudaGetLastError();
}

}  // namespace heat
