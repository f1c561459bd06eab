// Batched FP64 EMD sift for sm_100a -- the hot path behind GPUBatchEMD.
//
// Behaviour follows the reference's emd_batch_kernel (SeismicFlow/emd-cuda,
// kernels.py:834-1080) and its device functions, re-built for B200:
//
//  * one CTA (128, 256 or 512 threads) per trace, persistent: CTAs pull trace tickets from an
//    atomic work queue (FIFO, or a caller-given order), so a long trace never
//    holds a wave back and CSR batches of mixed length run in one launch;
//  * the proto-IMF lives in shared memory for the whole decomposition; the
//    running residue lives in the output rows (each row is written once, the
//    residue row once more per IMF);
//  * extrema: one warp-contiguous scan per sift pass computes ballot masks,
//    zero-crossing counts and the serial-fallback trigger; the masks are
//    compacted (popc ranks) straight into both envelopes' knot arrays, and
//    their prefix counts give every sample its knot segment in O(1) when the
//    knot list is strictly increasing (the reference binary-searches,
//    kernels.py:722-726).  The post-update scan of pass n is reused as the
//    pre-scan of pass n+1 (the reference scans the same data twice,
//    kernels.py:930 vs 965);
//  * boundary mirroring runs on one warp, eight lanes to each mirrored end;
//  * the upper and lower not-a-knot systems are solved concurrently by
//    parallel cyclic reduction (ping-pong buffers, one barrier per level), and
//    levels that can no longer change a bit are left out;
//  * envelope evaluation, the mean update and the six stop-test partial
//    sums are one fused pass; sums are formed in the reference's order (128
//    strided lanes + halving tree) and this file is compiled with
//    -fmad=false, so every value equals the reference algorithm's FP64
//    result bit for bit (the CPU oracle checks this);
//  * every quotient is the IEEE one, but those of the hot loops are formed
//    without the division's slow-path branch, by Markstein corrections from a
//    reciprocal (one correction is exact for the integer operands of the
//    integer time axis) or the approximate one (the PCR rows); a vote per
//    pass makes sure that their operands are in the exact ranges, and other
//    passes divide;
//  * one trace's pass is a chain of short phases between barriers, four
//    traces share an SM, and the code of a pass is as large as the 32 KB
//    instruction cache (straight-line code past 2048 instructions runs at half
//    the rate here with 16 warps): loops are kept rolled, rare paths are out
//    of line with one call site each, and range tests are taken out of loops.
//
// Per-pass knot/PCR storage is placed by size: all in the CTA's shared-
// memory arena; "borrow" (the proto-IMF parked in the per-CTA global slab
// during the spline solve so both PCR buffers stay on-chip, or with the
// moments beside the knots when the arena is short); "split" (PCR
// buffer 1 in the slab); "park" (the proto-IMF parked, PCR buffer 1 in its
// place, the knots and buffer 0 in the slab); or all in the slab.  For the
// host pipeline the kernel also reports finished chunks of traces through
// flags in mapped host memory.  Nothing here waits on another CTA or on the
// host.

#include "emdb_internal.cuh"

// Settled when the passes were longer (16,384 x 2048 seismic took 79 ms, now 53):
// one sift-pass instance for the on-chip placements and one for the off-chip
// ones (208.4k signals/s; one instance for all 195.6k, one per placement 184.9k),
// the six end-of-pass trees spread over the warps (188.1k on one warp):
// instruction supply decides as much as FP64 latency.
// Tuning knobs (compile-time; results are identical for every setting):
//  EMDB_LANE_UNROLL  wide instances: unroll factor of the lane-sum loops (the
//                  loads of a lane's samples in flight at once).  With the
//                  six sums split over the 128-lane groups, B200, 512 threads
//                  1024 x 8192 seismic / 256 threads 2048 x 4096 (ms): 4: 145.5 /
//                  47.8, 8: 143.0 / 47.4, 16: 142.5 / 47.3.
#ifndef EMDB_LANE_UNROLL
#define EMDB_LANE_UNROLL 16
#endif
//  EMDB_LOAD_CLOCKS  instrumented build: thread 0 of each CTA adds the clock64
//                  cycles of every trace's load into shared memory, of the
//                  whole trace, and of each phase of the sift passes (taken at
//                  the barriers that end them) to the plan's counters [2..]
//                  (emdb_plan_phase_clocks); off in the product build
#ifndef EMDB_LOAD_CLOCKS
#define EMDB_LOAD_CLOCKS 0
#endif
#if EMDB_LOAD_CLOCKS
// phases: 0 knot fill, 1 mirroring (+ parking), 2 spline rows, 3 PCR levels,
// 4 diagonal solve, 5 evaluation / update, 6 lane sums, 7 reduction trees +
// extrema scan, 8 per-IMF rows and reload, 9 the rest of the loop
#define EMDB_PH(Cptr, k)                                      \
  do {                                                        \
    if (threadIdx.x == 0) {                                   \
      const long long t_ = clock64();                         \
      (Cptr)->ph[k] += (unsigned long long)(t_ - (Cptr)->ph_last); \
      (Cptr)->ph_last = t_;                                   \
    }                                                         \
  } while (0)
#else
#define EMDB_PH(Cptr, k) do {} while (0)
#endif
constexpr int kPhases = 10;

// EMDB_F32: the FP32 build of this file (namespace emdb::f32).  Every value
// the sift computes is a `real`; the reference kernel's double literals keep
// their C++ meaning, so float expressions that mix them are evaluated in
// double and rounded once, as in the reference source compiled with REAL_T =
// float.  Its quotients (div_q from an IEEE reciprocal; on the integer axis quot
// and div_core from the approximate one) are self-tested against the float
// division by emdb_check_division modes 3, 4 and 6; the one double quotient per
// envelope sample (the reference's "/ 6.0") is formed from RN(1/6) and its
// residual (div6), which equals the double division.
#ifndef EMDB_F32
#define EMDB_F32 0
#endif
#if EMDB_F32
namespace emdb::f32 {
using real = float;
#else
namespace emdb {
using real = double;
#endif

namespace {

constexpr unsigned kFull = 0xffffffffu;

// two values loaded and stored as one word
struct alignas(2 * sizeof(real)) real2 { real x, y; };

constexpr int kLaneUnroll = EMDB_LANE_UNROLL;

// reference thresholds (kernels.py:81-85, 814, 1069): the first five are
// REAL_T functions there, the last two double literals compared with REAL_T
constexpr real kEnergyRatioThr = 0.2;
constexpr real kStdThr = 0.2;
constexpr real kSvarThr = 0.001;
constexpr real kTotalPowerThr = 0.005;
constexpr real kRangeThr = 0.001;
constexpr double kSumNewSqMin = 1e-10;
constexpr double kResidueZeroAtol = 1e-8;
constexpr int kLocalExtBuf = 64;  // kernels.py:206 (serial-fallback trigger)

struct Ctl {
  int job;
  int head[2][kMaxNbsym + 1];  // first NB+1 extrema indices per side (0 = max, 1 = min)
  int tail[2][kMaxNbsym + 1];  // tail[q][k] = index of extremum n_q-1-k
  int zero_first;              // the scanned trace starts with a zero (N > kFallbackFrom)
  int unused[39];              // keeps the block's size: it decides the longest trace a CTA takes
  int lsym, rsym;
  int kbase[2], kcnt[2];
  int dbg_n[kMaxImfsCap], dbg_e[kMaxImfsCap], dbg_z[kMaxImfsCap];
  int chunk_bad;
  real sums[8];
#if EMDB_LOAD_CLOCKS
  unsigned long long ph[kPhases];
  long long ph_last;
#endif
};

// The 6 x 128 reduction lanes have no fixed home: between sift passes they sit
// at the start of the knot arena; inside a pass, after the spline solve, they
// reuse PCR buffer 1, which is dead from then on (or follow the PCR buffers
// when those are smaller than the lanes).
constexpr int kRedDoubles = 6 * kThreads;
constexpr size_t kRedBytes = kRedDoubles * sizeof(real);

// Extrema-scan slots of a CTA of NT threads: one contiguous range of 32-sample
// chunks per slot, scanned by one warp and filled into knots by one warp.
template <int NT>
__host__ __device__ constexpr int scan_slots() {
  return NT / 32;
}

// Per-warp scan counts live right after the control block, one 16-byte word a
// warp: maxima | minima << 16, sign changes, zero-run ends, fallback trigger
// (room for 5 ints a warp).
struct SmemLayout {
  Ctl* ctl;
  uint4* wc;          // [NW]
  real* red;        // [6][128] between passes (= arena start)
  real* imf;        // [N]
  uint2* mm;          // [nch] ballot masks of the last extrema scan: maxima, minima
  uint32_t* pp;       // per-chunk exclusive prefixes within the owning warp's range:
                      // maxima | minima << 16 (the fill makes them global)
  char* arena;        // knot arena start
  int arena_bytes;    // bytes left for the knot arena
};

// sizes: size_t on the host (a query must not wrap for any int input), 32 bits
// in the kernel, where the launch has checked that they fit
#ifdef __CUDA_ARCH__
using usize = unsigned;
#else
using usize = size_t;
#endif
__host__ __device__ inline usize align16(usize x) { return (x + 15) & ~usize(15); }

// NT: threads per CTA (128, or 512 for the wide instance).  kGImf: the
// proto-IMF lives in the CTA's global slab instead of shared memory (traces
// longer than shared memory holds); it then takes no shared memory.
template <int NT = kThreads, bool kGImf = false>
__host__ __device__ inline usize fixed_bytes(int N) {
  usize nch = (usize)(N + 31) / 32;
  usize b = align16(sizeof(Ctl)) + align16(5 * (NT / 32) * sizeof(int));
  if (!kGImf) b += align16((usize)N * sizeof(real));
  b += align16(nch * 4) * 2 + align16(nch * 2) * 2;
  return b;
}

template <int NT = kThreads, bool kGImf = false>
__device__ __forceinline__ SmemLayout carve(char* base, int N, int arena_total,
                                            real* gimf = nullptr) {
  SmemLayout L;
  usize nch = (usize)(N + 31) / 32;
  char* p = base;
  L.ctl = reinterpret_cast<Ctl*>(p); p += align16(sizeof(Ctl));
  L.wc = reinterpret_cast<uint4*>(p); p += align16(5 * (NT / 32) * sizeof(int));
  L.mm = reinterpret_cast<uint2*>(p); p += align16(nch * 4) * 2;
  L.pp = reinterpret_cast<uint32_t*>(p); p += align16(nch * 2) * 2;
  // the proto-IMF directly ahead of the arena: the borrow placement uses both
  // as one region
  if (kGImf) {
    L.imf = gimf;
  } else {
    L.imf = reinterpret_cast<real*>(p); p += align16((usize)N * sizeof(real));
  }
  L.arena = p;
  L.red = reinterpret_cast<real*>(p);
  L.arena_bytes = arena_total - (int)(p - base);
  return L;
}

// Knot / PCR storage for one sift pass (both envelopes).  A PCR buffer holds
// blocks of eight rows: their (a, c) pairs, then their (b, d) pairs, so one
// address serves both halves of a row and eight consecutive rows of either
// half cover all banks once.  It has room for `cap` rows; the two systems take
// at most cap - 8 (an envelope has at most its extrema plus 2 nbsym knots),
// which leaves a row for the neighbour of rows that have none and the last
// block's padding.  The spline moments M take the place of buffer 0, whose
// rows nothing reads any more by then.
struct Knots {
  real2* XY[2]; // (position, value) of each knot
  real* M[2];
  real* P[2];   // ping-pong PCR buffers, each `cap` rows
  real* red;    // reduction lanes after the solve: buffer 1, or just past it
  int cap;
  __device__ __forceinline__ char* rows(int q) const {
    return reinterpret_cast<char*>(q ? P[1] : P[0]);
  }
};

__host__ __device__ inline usize knot_bytes(int kc0, int kc1) {
  // usize throughout: a host-side size query must not wrap for any int input
  const usize cap = (usize)kc0 + (usize)kc1;
  const usize red_extra = (4 * cap >= (usize)kRedDoubles) ? 0 : kRedBytes;
  return (2 * cap + 8 * cap) * sizeof(real) + red_extra;
}

__device__ __forceinline__ Knots place_knots(char* base, int kc0, int kc1) {
  Knots K;
  real* p = reinterpret_cast<real*>(base);
  K.XY[0] = reinterpret_cast<real2*>(p);
  K.XY[1] = K.XY[0] + kc0;
  p += 2 * (kc0 + kc1);
  K.cap = kc0 + kc1;
  K.P[0] = p; p += 4 * K.cap;
  K.P[1] = p;
  K.M[0] = K.P[0];
  K.M[1] = K.P[0] + kc0;
  K.red = (4 * K.cap >= kRedDoubles) ? K.P[1] : K.P[1] + 4 * K.cap;
  return K;
}

// Split placement, for passes whose knots fit shared memory only without the
// second PCR buffer: knots X | Y and PCR buffer 0 (which ends up holding the
// moments) in the arena, buffer 1 in the per-CTA global slab.  Evaluation then
// reads shared memory only, and half of the PCR levels read the slab.
__host__ __device__ inline usize split_bytes(int kc0, int kc1) {
  return 6 * ((usize)kc0 + (usize)kc1) * sizeof(real);
}

__device__ __forceinline__ Knots place_knots_split(char* sbase, int sbytes, char* gbase, int kc0,
                                                   int kc1) {
  Knots K;
  real* p = reinterpret_cast<real*>(sbase);
  K.XY[0] = reinterpret_cast<real2*>(p);
  K.XY[1] = K.XY[0] + kc0;
  p += 2 * (kc0 + kc1);
  K.cap = kc0 + kc1;
  K.P[0] = p; p += 4 * K.cap;
  K.P[1] = reinterpret_cast<real*>(gbase);
  K.M[0] = K.P[0];
  K.M[1] = K.P[0] + kc0;
  // reduction lanes: shared memory past buffer 0 when they fit, else the slab
  // (buffer 1 is dead after the solve; the slab holds knot_bytes of the largest pass)
  if (split_bytes(kc0, kc1) + kRedBytes <= (usize)sbytes) K.red = p;
  else K.red = (4 * K.cap >= kRedDoubles) ? K.P[1] : K.P[1] + 4 * K.cap;
  return K;
}

// Borrow placement, for passes whose knots fit shared memory only together
// with the proto-IMF's space: the proto-IMF is parked in the per-CTA slab
// during the solve, PCR buffer 1 takes its place (imf region plus the arena
// ahead of the knots), and X | Y | buffer 0 sit at the end of the arena, clear
// of the proto-IMF that the knot fill reads.  Evaluation reads the old sample
// values back from the slab; the reduction lanes go to the slab after them.
__host__ __device__ inline bool borrow_fits(int N, int arena_bytes, usize slab_stride, int kc0,
                                            int kc1) {
  const usize cap = (usize)kc0 + (usize)kc1;
  const usize region = align16((usize)N * sizeof(real)) + (usize)arena_bytes;
  return 6 * cap * sizeof(real) <= (usize)arena_bytes &&
         10 * cap * sizeof(real) <= region &&
         (align16((usize)N * sizeof(real)) + kRedBytes) <= slab_stride;
}

__device__ __forceinline__ real* borrow_save(char* slab) { return reinterpret_cast<real*>(slab); }

__device__ __forceinline__ Knots place_knots_borrow(real* imf, char* arena, int arena_bytes,
                                                    char* slab, int N, int kc0, int kc1) {
  Knots K;
  K.cap = kc0 + kc1;
  real* p = reinterpret_cast<real*>(arena + arena_bytes) - 6 * K.cap;
  K.XY[0] = reinterpret_cast<real2*>(p);
  K.XY[1] = K.XY[0] + kc0;
  p += 2 * (kc0 + kc1);
  K.P[0] = p;
  K.P[1] = imf;
  K.M[0] = K.P[0];
  K.M[1] = K.P[0] + kc0;
  K.red = reinterpret_cast<real*>(slab + align16((usize)N * sizeof(real)));
  return K;
}

// Compact borrow placement, for long traces whose X | Y | buffer 0 do not fit
// the arena next to the proto-IMF: the moments get their own array beside the
// knots (instead of buffer 0's dead a / c arrays), so only X | Y | M sit at the
// arena's end and both PCR buffers go to the front of the proto-IMF region
// (parked in the slab, as for the borrow placement).  Everything stays
// on-chip; the arena needs 3 doubles per knot slot instead of 6, the region
// 11 instead of 10.
__host__ __device__ inline bool borrow2_fits(int N, int arena_bytes, usize slab_stride, int kc0,
                                             int kc1) {
  const usize cap = (usize)kc0 + (usize)kc1;
  const usize region = align16((usize)N * sizeof(real)) + (usize)arena_bytes;
  return 3 * cap * sizeof(real) <= (usize)arena_bytes &&
         11 * cap * sizeof(real) <= region &&
         (align16((usize)N * sizeof(real)) + kRedBytes) <= slab_stride;
}

__device__ __forceinline__ Knots place_knots_borrow2(real* imf, char* arena, int arena_bytes,
                                                     char* slab, int N, int kc0, int kc1) {
  Knots K;
  K.cap = kc0 + kc1;
  real* p = reinterpret_cast<real*>(arena + arena_bytes) - 3 * K.cap;
  K.M[0] = p;
  K.M[1] = p + kc0;
  p += K.cap;         // the pairs last: 16-byte aligned whatever the knot count
  K.XY[0] = reinterpret_cast<real2*>(p);
  K.XY[1] = K.XY[0] + kc0;
  K.P[0] = imf;
  K.P[1] = imf + 4 * K.cap;
  K.red = reinterpret_cast<real*>(slab + align16((usize)N * sizeof(real)));
  return K;
}

// Park placement, for passes whose knots fit neither shared-memory placement
// but whose PCR buffer 1 fits the proto-IMF's space (long traces with many
// knots): the proto-IMF is parked in the slab as for the borrow placement,
// buffer 1 takes its place (imf region plus the arena ahead), and X | Y |
// buffer 0 go to the slab after the parked samples.  Half of the PCR levels
// then read shared memory; the evaluation reads the knots and the old samples
// from the slab.  The reduction lanes use the arena start, free after the
// solve.
__host__ __device__ inline bool park_fits(int N, int arena_bytes, usize slab_stride, int kc0,
                                          int kc1) {
  const usize cap = (usize)kc0 + (usize)kc1;
  const usize imfb = align16((usize)N * sizeof(real));
  return 4 * cap * sizeof(real) <= imfb + (usize)arena_bytes &&
         imfb + 6 * cap * sizeof(real) <= slab_stride;
}

__device__ __forceinline__ Knots place_knots_park(real* imf, char* slab, int N, int kc0, int kc1,
                                                  real* red) {
  Knots K;
  K.cap = kc0 + kc1;
  real* p = reinterpret_cast<real*>(slab + align16((usize)N * sizeof(real)));
  K.XY[0] = reinterpret_cast<real2*>(p);
  K.XY[1] = K.XY[0] + kc0;
  p += 2 * (kc0 + kc1);
  K.P[0] = p;
  K.P[1] = imf;
  K.M[0] = K.P[0];
  K.M[1] = K.P[0] + kc0;
  K.red = red;
  return K;
}

enum : int { kPlaceSmem = 0, kPlaceSplit = 1, kPlaceSlab = 2, kPlaceBorrow = 3, kPlacePark = 4,
              kPlaceBorrow2 = 5 };
enum : int { kOnChip = -1, kOffChip = -2, kAnyPlace = -3 };

// Where one sift pass keeps its knots and PCR buffers: the first placement
// that fits, the on-chip ones first (shared, borrow, compact borrow), then
// split, park, slab.  `arena_bytes` is the knot arena left after the fixed
// part (control block, scan masks, proto-IMF); the slab always fits.
__host__ __device__ inline int choose_place(int N, int arena_bytes, usize slab_stride, int kc0,
                                            int kc1, bool imf_global = false) {
  // a proto-IMF in global memory has no shared-memory region to lend: only
  // the placements that leave it alone
  if (imf_global)
    return knot_bytes(kc0, kc1) <= (usize)arena_bytes ? kPlaceSmem
         : split_bytes(kc0, kc1) <= (usize)arena_bytes ? kPlaceSplit
                                                        : kPlaceSlab;
  return knot_bytes(kc0, kc1) <= (usize)arena_bytes ? kPlaceSmem
       : borrow_fits(N, arena_bytes, slab_stride, kc0, kc1) ? kPlaceBorrow
       : borrow2_fits(N, arena_bytes, slab_stride, kc0, kc1) ? kPlaceBorrow2
       : split_bytes(kc0, kc1) <= (usize)arena_bytes ? kPlaceSplit
       : park_fits(N, arena_bytes, slab_stride, kc0, kc1) ? kPlacePark
                                                          : kPlaceSlab;
}

// Correctly rounded a/b from y = RN(1/b) (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 1990):
// if y is within half an ulp of 1/b and q within one ulp of a/b, then with the
// exact remainder r = a - b*q (one FMA), RN(q + r*y) = RN(a/b).  q0 = RN(a*y)
// can be 1.5 ulp off, so one correction step first brings it within one ulp,
// the second rounds correctly.  Operands whose remainders or quotient could
// underflow or overflow (|a| or |a*y| outside [2^-900, 2^900], zeros, inf,
// NaN) take the division.
// A zero numerator gives q0 = a*y, the correctly signed zero (or NaN when y is
// infinite or NaN, as a/b would be).  Checked bit for bit against the hardware
// division by emdb_check_division.
//
__device__ __noinline__ double div_slow(double a, double b) { return a / b; }

#if EMDB_F32
// Float counterpart: div_q is the two-step Markstein quotient from y = RN(1/b)
// (Muller et al., Handbook of Floating-Point Arithmetic, ch. 4.9 / 5.3).  `slow`
// is set outside the ranges where every step is exact: |a|, |q| in
// (2^-100, 2^100).
__device__ __noinline__ float div_slow(float a, float b) { return a / b; }

__device__ __forceinline__ float div_q(float a, float b, float y, bool& slow) {
  const float q0 = a * y;
  const float e0 = fmaf(-q0, b, a);
  const float q1 = fmaf(e0, y, q0);
  const float e1 = fmaf(-q1, b, a);
  const float q2 = fmaf(e1, y, q1);
  const float aa = fabsf(a), qa = fabsf(q0);
  const bool zero = a == 0.0f;
  slow |= !(zero || (aa > 0x1p-100f && aa < 0x1p+100f && qa > 0x1p-100f && qa < 0x1p+100f));
  return zero ? q0 : q2;
}

// 1/b within (1/2 + 2^-21) ulp, and a/b from it: the argument is the one at the
// FP64 div_core, with 24 bits for 53.  y's relative error is at most
// (1 + 2^-20) 2^-25 m_b (m_b in [1, 2) the significand of b) and the remainder
// half an ulp of q, so the last step is off by less than the 2^-24 / m_b ulp(q)
// that separate a quotient from a rounding boundary when m_b < 2 - 2^-18; the
// 64 significands nearest 2 are checked with every numerator
// (emdb_check_division mode 3, like all integer pairs up to 65536).  The
// remainders are exact for |a| >= 2^-102 and |b| in [2^-5, 2^24), where q is
// normal too.
__device__ __forceinline__ float recip(float h) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(h));
  return fmaf(fmaf(-h, y, 1.0f), y, y);
}
__device__ __forceinline__ float quot(float a, float h, float y) {
  float q = a * y;
  q = fmaf(fmaf(-q, h, a), y, q);
  return fmaf(fmaf(-q, h, a), y, q);
}

__device__ __forceinline__ float div_core(float a, float b) { return quot(a, b, recip(b)); }
// neither zero nor at least 2^-80
__device__ __forceinline__ bool tiny(float x) {
  return (__float_as_uint(x) & 0x7fffffffu) - 1u < (47u << 23) - 1u;
}
#endif

// The two corrections without the tests, for a numerator of zero or in range
// (a negative zero gives +0).
__device__ __forceinline__ double quot(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-q, b, a), y, q);
  return fma(fma(-q, b, a), y, q);
}

#if !EMDB_F32
// Branch-free RN(a/b) with no reciprocal at hand (FMA division schemes of
// Markstein, IBM J. Res. Dev. 1990, and Muller et al., "Handbook of
// Floating-Point Arithmetic", 2nd ed., ch. 4.7): y from the PTX approximate
// reciprocal, one cubic step (1/b = y(1 + e + e^2 + ...), e = 1 - by) and one
// linear one, whose argument is within 2^-104 of 1/b before its rounding, so y
// is within (1/2 + 2^-51) ulp of it; q1 = RN(q0 + (a - b q0) y) is then within
// (1/2 + 2^-50) ulp of a/b, its remainder r = a - b q1 exact, and q1 + r y
// differs from a/b by at most |r/b| times y's relative error, below
// 2^-55 m_b ulp(q) (m_b in [1, 2) the significand of b; the 2^-51 adds nothing
// that matters: for m_b = 2 - 2^-52 y's error is at most half an ulp of 1/b
// to within 2^-53).  A quotient of 53-bit numbers is never closer than
// 2^-53 / m_b ulp(q) to a rounding boundary without lying on it, and never
// lies on it, so the last FMA rounds as the division does.
//
// div_nb, the form that emdb_check_division tests, sets `slow` unless |a|, |b|
// and |q| are in [2^-511, 2^512), where no step underflows or overflows:
// exponent fields 512..1535 are those whose two top bits differ, i.e. whose
// high word plus 2^29 has bit 30 set.  The PCR rows make sure of their
// operands beforehand (solve_splines).
// 10 FP64 operations; the form before it (two linear steps, a neighbour choice
// by two exact remainders and range compares on the doubles) took 8 and 11
// compares, which cost as much as arithmetic.
__device__ __forceinline__ unsigned range_bits(double x) {
  return (unsigned)__double2hiint(x) + 0x20000000u;
}
// 1/b to within (1/2 + 2^-51) ulp; RN(1/b) for an integer b up to 65536, which
// is never that close to the middle of two doubles (checked for each by
// emdb_check_division mode 0).
__device__ __forceinline__ double recip(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  double e = fma(-b, y, 1.0);
  e = fma(e, e, e);
  y = fma(e, y, y);
  e = fma(-b, y, 1.0);
  return fma(e, y, y);
}
// The quotient without its range checks (+0 for any zero numerator).
__device__ __forceinline__ double div_core(double a, double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  double e = fma(-b, y, 1.0);
  e = fma(e, e, e);
  y = fma(e, y, y);
  const double q0 = a * y;
  e = fma(-b, y, 1.0);
  y = fma(e, y, y);
  const double r0 = fma(-q0, b, a);
  const double q1 = fma(r0, y, q0);
  const double r1 = fma(-q1, b, a);
  return fma(r1, y, q1);
}
__device__ __forceinline__ double div_nb(double a, double b, bool& slow) {
  const double q = div_core(a, b);
  slow |= !(range_bits(a) & range_bits(b) & range_bits(q) & 0x40000000u);
  return q;
}
#endif
// high word of |x|: orders magnitudes, and (as a fixed-point number with 20
// fraction bits) is within 0.0861 below log2|x| plus the exponent bias
__device__ __forceinline__ unsigned mag(double x) {
  return (unsigned)__double2hiint(x) & 0x7fffffffu;
}
__device__ __forceinline__ unsigned mag(float x) {
  return (unsigned)__float_as_int(x) & 0x7fffffffu;
}

#if !EMDB_F32
// with the tests, for emdb_check_division
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  const double q = quot(a, b, y), aa = fabs(a), qa = fabs(q);
  if (a == 0.0) return a * y;
  const bool in = aa > 0x1p-900 && aa < 0x1p+900 && qa > 0x1p-900 && qa < 0x1p+900;
  return in ? q : div_slow(a, b);
}
#endif

// RN(x / 6) for the spline term (kernels.py:733) in two operations: with
// 1/6 = C + c, C = RN(1/6), the product x*C plus the rounded correction x*c is
// within 2^-104 |x/6| of x/6 before its one rounding (multiplication by a
// constant held as two words: Brisebarre and Muller, IEEE Trans. Computers
// 57(2), 2008), and x/6 is never closer than a sixth of its ulp u to a
// rounding boundary m: x is a multiple of 4u and 6m an odd multiple of u, so
// |x - 6m| >= u.  `slow` is set for a non-zero x outside
// [2^-900, 2^900) (subnormal products, infinities, NaN).  Checked against the
// division by emdb_check_division mode 1.
constexpr double kInv6 = 1.0 / 6.0;
constexpr double kInv6Lo = kInv6 / 18014398509481984.0;   // RN(1/6 - RN(1/6)) = RN(1/6) / 2^54
__device__ __forceinline__ bool odd_range(double x) {
  const unsigned v = (unsigned)__double2hiint(x) & 0x7fffffffu;
  // exponents [-900, 900): biased 123..1922
  return (v - (123u << 20)) >= (1800u << 20) && (v | (unsigned)__double2loint(x)) != 0u;
}
__device__ __forceinline__ double div6(double x) { return fma(x, kInv6, x * kInv6Lo); }
__device__ __forceinline__ double div6(double x, bool& slow) {
  slow |= odd_range(x);
  return div6(x);
}
// a moment that is neither zero nor in [2^-700, 2^900) (biased exponents 323..1922)
__device__ __forceinline__ bool odd_moment(double m) {
  const unsigned v = (unsigned)__double2hiint(m) & 0x7fffffffu;
  return v - (323u << 20) >= (1600u << 20) && (v | (unsigned)__double2loint(m)) != 0u;
}

// longest integer segment that eval_seg_int takes
constexpr int kMaxIntSeg = 65536;

struct TimeAxis {
  const real* T;
  bool arange;
  __device__ __forceinline__ real operator()(int i) const { return arange ? (real)i : T[i]; }
};

// ---------------------------------------------------------------------------
// Extrema: count pass (find_extrema_parallel semantics, kernels.py:231-349,
// with the serial scan's plateau rule, kernels.py:157-200).
// ---------------------------------------------------------------------------
// Longest trace whose zero-crossing count no chunk fallback can change
constexpr int kFallbackFrom = kThreads * 128;

// NS slots; `slot` is the calling warp's slot.
//
// The common chunk has no flat step, no exact zero and no underflowing product
// in it or just before it; there an extremum is dp*dn < 0, its kind the sign
// bit of dp, and a crossing v*vn < 0, four compares of doubles a sample in all
// (all the reference's tests, kernels.py:157-200, took ten).  Any sample that
// could be otherwise (a product that is zero or NaN) sends its chunk, and the
// next one, whose first sample looks back at it, through those tests.
// Neighbours come straight from shared memory (conflict-free consecutive
// words): no shuffles, iterations independent.  Two chunks a trip where one
// trace has an SM to itself, one where four share it (16,384 x 2048 seismic
// 71.9 ms at one, 73.8 at two; 256 x 8192 65.0 and 64.6).
template <int NS>
__device__ __forceinline__ void extrema_count(const SmemLayout& L, int N, int slot, int lane) {
  const real* imf = L.imf;
  const int nch = (N + 31) >> 5;
  const int c0 = (slot * nch) / NS, c1 = ((slot + 1) * nch) / NS;
  uint32_t run = 0;              // maxima | minima << 16 of the slot so far
  int zc = 0, zre = 0;
  bool trig = false;
  bool careful = c0 > 0 && c0 < c1 && imf[(c0 << 5) - 1] == real(0);
#pragma unroll (NS == kWarps ? 1 : 2)
  for (int c = c0; c < c1; ++c) {
    const int i = (c << 5) + lane;
    const real v = imf[min(i, N - 1)], vp = imf[max(min(i, N) - 1, 0)], vn = imf[min(i + 1, N - 1)];
    const bool interior = i >= 1 && i <= N - 2, left = i <= N - 2;
    const real dp = v - vp, dn = vn - v;
    const real turn = dp * dn, cross = v * vn;
    const bool strict = interior && turn < real(0);
    bool ismin = strict && dp < real(0);
    bool ismax = strict && !(dp < real(0));
    const bool sc = left && cross < real(0);
    const bool odd = (interior && !(fabs(turn) > real(0))) || !(fabs(cross) > real(0));
    const bool any_odd = __any_sync(kFull, odd);
    if (any_odd || careful) {
      if (interior && dn == real(0) && dp != real(0)) {
        // rare: true left edge of a flat run, classified by the slopes around it
        int j = i;
#pragma unroll 1
        while (j + 1 < N && imf[j + 1] == v) ++j;
        if (j + 1 < N) {
          const real da = imf[j + 1] - imf[j];
          if (dp > real(0) && da < real(0)) ismax = true;
          else if (dp < real(0) && da > real(0)) ismin = true;
        }
      }
      trig |= interior && (dp == real(0) || dn == real(0) || v == real(0));
      const bool zr = i >= 1 && i < N && v != real(0) && vp == real(0);
      zre += __popc(__ballot_sync(kFull, zr));
    }
    careful = any_odd;
    const uint32_t bmax = __ballot_sync(kFull, ismax);
    const uint32_t bmin = __ballot_sync(kFull, ismin);
    if (lane == 0) {
      L.mm[c] = make_uint2(bmax, bmin);
      L.pp[c] = run;
    }
    run += (uint32_t)__popc(bmax) + ((uint32_t)__popc(bmin) << 16);
    zc += __popc(__ballot_sync(kFull, sc));
  }
  trig = __any_sync(kFull, trig);
  if (lane == 0) L.wc[slot] = make_uint4(run, (uint32_t)zc, (uint32_t)zre, trig ? 1u : 0u);
}

struct ExtInfo {
  int n_max, n_min;       // stored (capped) counts
  int n_zer;
  uint32_t off;           // this warp's rank offsets: maxima | minima << 16
  bool overflow;
  bool trig;              // serial-fallback trigger (exact zeros / flat runs)
};

// After the count pass + barrier.  Reproduces the parallel/serial split of
// find_extrema_parallel: without a fallback trigger the zero-crossing count is
// sign changes only; with one, the serial count adds one per zero run that
// ends before N (kernels.py:123-143, 273-276).
// One lane reads one warp's word; a warp then sums them (the counts of a kind
// are below 2^16 for the longest trace).  `warp`: the caller's, for its rank
// offsets.
template <int NS>
__device__ __forceinline__ ExtInfo extrema_totals(const SmemLayout& L, int warp, int lane,
                                                  int max_extrema) {
  const uint4 w = lane < NS ? L.wc[lane] : make_uint4(0u, 0u, 0u, 0u);
  const uint32_t tot = __reduce_add_sync(kFull, w.x);
  const uint32_t zc = __reduce_add_sync(kFull, w.y);
  ExtInfo e;
  e.off = __reduce_add_sync(kFull, lane < warp ? w.x : 0u);
  e.trig = __any_sync(kFull, w.w != 0u);
  e.n_zer = (int)zc;
  if (e.trig || L.ctl->chunk_bad) e.n_zer += (int)__reduce_add_sync(kFull, w.z);
  const int tot_max = (int)(tot & 0xffffu), tot_min = (int)(tot >> 16);
  e.n_max = min(tot_max, max_extrema);
  e.n_min = min(tot_min, max_extrema);
  e.overflow = tot_max >= max_extrema || tot_min >= max_extrema;
  return e;
}

// The reference's parallel scan also falls back when one thread's contiguous
// chunk (ceil(N/128) samples) holds more than 64 strict maxima or minima.  That
// can only change n_zer when imf[0] == 0 (leading zero), and only for N > 16384,
// so it is evaluated in that rare case only.  The chunks are the reference's
// 128 threads' (threads past 128 of a wider CTA have none).  Ends with a barrier.
__device__ void chunk_fallback_check(const SmemLayout& L, int N, int tid) {
  Ctl& C = *L.ctl;
  const real* s = L.imf;
  int cs = (N + kThreads - 1) / kThreads;
  int start = tid * cs, end = min(start + cs, N);
  int lo = max(start, 1), hi = min(end, N - 1);
  int nmx = 0, nmn = 0;
#pragma unroll 1
  for (int i = lo; i < hi; ++i) {
    real dp = s[i] - s[i - 1], dn = s[i + 1] - s[i];
    if (dp * dn < 0.0) { if (dp < 0.0) ++nmn; else ++nmx; }
  }
  int bad = __syncthreads_or(nmx > kLocalExtBuf || nmn > kLocalExtBuf);
  if (tid == 0) C.chunk_bad = bad;
  __syncthreads();
}

// One extrema scan = count pass + totals, and the reference's rare chunk
// fallback.  Ends after a barrier with every thread holding the same totals
// and its warp's rank offsets.  Nothing here reads imf[] after the last
// barrier: the caller may write it at once (the emission of a row does), and a
// warp that came late to a test on imf[] would enter the fallback's barriers
// alone.  So thread 0 looks at the first sample before it.
template <int NT>
__device__ __forceinline__ ExtInfo extrema_scan(const SmemLayout& L, int N, int tid, int warp,
                                                int lane, int max_extrema) {
  constexpr int NS = scan_slots<NT>();
  extrema_count<NS>(L, N, warp, lane);
  if (tid == 0) {
    L.ctl->chunk_bad = 0;
    if (N > kFallbackFrom) L.ctl->zero_first = L.imf[0] == real(0);
  }
  __syncthreads();
  ExtInfo e = extrema_totals<NS>(L, warp, lane, max_extrema);
  if (N > kFallbackFrom && L.ctl->zero_first && !e.trig) {
    chunk_fallback_check(L, N, tid);
    e = extrema_totals<NS>(L, warp, lane, max_extrema);
  }
  return e;
}

// ---------------------------------------------------------------------------
// Knot fill: compacted true extrema -> X/Y at offset NB (both sides).
// Returns this thread's "bad envelope sign" vote for true knots.
// ---------------------------------------------------------------------------
// NS slots; the calling warp fills slot `warp` (warps past NS do not call it)
template <int NS>
__device__ __forceinline__ bool fill_true_knots(const SmemLayout& L, const Knots& K,
                                                const ExtInfo& e, int N, int NB,
                                                const TimeAxis& T, int warp, int lane) {
  Ctl& C = *L.ctl;
  const real* imf = L.imf;
  int nch = (N + 31) >> 5;
  int c0 = (warp * nch) / NS, c1 = ((warp + 1) * nch) / NS;
  unsigned lt = (1u << lane) - 1u;
  bool bad = false;
  const int off_max = (int)(e.off & 0xffffu), off_min = (int)(e.off >> 16);
  // one extremum lane: rank it, write its knot, note head / tail indices
  auto put = [&](uint32_t bm, uint32_t bn, int pm, int pn, int ii, real v) {
    const bool ismax = (bm >> lane) & 1u;
    int q = ismax ? 0 : 1;
    int rank = q == 0 ? off_max + pm + __popc(bm & lt) : off_min + pn + __popc(bn & lt);
    int nq = q == 0 ? e.n_max : e.n_min;
    if (rank < nq) {
      (q == 0 ? K.XY[0] : K.XY[1])[NB + rank] = real2{T(ii), v};
      bad |= q == 0 ? (v < 0.0) : (v > 0.0);
      if (rank <= NB) C.head[q][rank] = ii;
      int fe = nq - 1 - rank;
      if (fe <= NB) C.tail[q][fe] = ii;
    }
  };
#pragma unroll (NS == kWarps ? 1 : 2)
  for (int c = c0; c < c1; ++c) {
    const uint2 m = L.mm[c];
    const uint32_t pp = L.pp[c];
    if (((m.x | m.y) >> lane) & 1u) {
      int ii = (c << 5) + lane;
      real v = imf[ii];
      if (e.trig) {
        // a proto-IMF with exact zeros or flat runs: a plateau extremum reports
        // the run's midpoint
        const real dp = v - imf[ii - 1], dn = imf[ii + 1] - v;
        if (!(dp * dn < 0.0)) {
          int j = ii;
#pragma unroll 1
          while (j + 1 < N && imf[j + 1] == v) ++j;
          ii = (ii + j) / 2;
          v = imf[ii];
        }
      }
      put(m.x, m.y, pp & 0xffff, pp >> 16, ii, v);
    }
  }
  // the chunks' prefixes become global (warp offset added) for the evaluation
  // pass's segment counts, once every lane has taken its ranks
  __syncwarp();
#pragma unroll 1
  for (int c = c0 + lane; c < c1; c += 32) L.pp[c] += e.off;
  return bad;
}

// ---------------------------------------------------------------------------
// Boundary mirroring (mirror_one_side, kernels.py:360-558) for both sides.
// Every lane of warp 0 makes the same O(1) decisions (which extremum comes
// first and last, whether the end sample lies beyond its neighbour, whether
// the mirrored knots reach the end) and then writes its own mirrored knots: a
// list is a run of extremum ranks plus possibly the end sample, so entry j
// needs no list in memory.  The chain is five dependent shared-memory reads;
// with the lists built by one lane, entry by entry, it was three to four times
// as long.  Knot positions are strictly increasing
// whenever T is (the host checks T), so the reference's adjacent-duplicate
// removal never drops a knot and is not needed here.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int ind_of(const Ctl& C, int q, int n, int NB, int k) {
  return k <= NB ? C.head[q][k] : C.tail[q][n - 1 - k];
}

// Ranks hi, hi-1, ..., lo of one kind of extremum; `end`: and the trace's end
// sample (on the left after them, on the right before them, the ranks then
// ascending).
struct MirrorList {
  int hi, lo, end;
  __device__ __forceinline__ int count() const { return max(hi - lo + 1, 0) + end; }
};

__device__ __forceinline__ bool mirror_both(const SmemLayout& L, const Knots& K, const ExtInfo& e,
                                            int N, int NB, const TimeAxis& T, int lane) {
  Ctl& C = *L.ctl;
  const real* S = L.imf;
  const int nM = e.n_max, nm = e.n_min;
  const int im0 = C.head[0][0], in0 = C.head[1][0], imL = C.tail[0][0], inL = C.tail[1][0];
  const real s0 = S[0], sN = S[N - 1];
  MirrorList l0, l1, r0, r1;
  int lsym, rsym;
  // ---- left bound: kernels.py:383-413 ----
  {
    const bool mf = im0 < in0;                       // a maximum comes first
    const real so = S[mf ? in0 : im0];
    const bool over = mf ? s0 > so : s0 < so;
    const int nf = mf ? nM : nm, no = mf ? nm : nM;
    const MirrorList f{min(nf, over ? NB + 1 : NB) - 1, over ? 1 : 0, 0};
    const MirrorList o{min(no, over ? NB : NB - 1) - 1, 0, over ? 0 : 1};
    l0 = mf ? f : o;
    l1 = mf ? o : f;
    lsym = over ? (mf ? im0 : in0) : 0;
  }
  // ---- right bound: kernels.py:415-454 ----
  {
    const bool mf = imL > inL;                       // a maximum comes last
    const real so = S[mf ? inL : imL];
    const bool over = mf ? sN > so : sN < so;
    const int nf = mf ? nM : nm, no = mf ? nm : nM;
    const MirrorList f{over ? nf - 2 : nf - 1, max(over ? nf - NB - 1 : nf - NB, 0), 0};
    const MirrorList o{no - 1, max(over ? no - NB : no - NB + 1, 0), over ? 0 : 1};
    r0 = mf ? f : o;
    r1 = mf ? o : f;
    rsym = over ? (mf ? imL : inL) : N - 1;
  }
  // An empty list falls back to the whole index list (kernels.py:456-459,
  // 523-531); that only happens when the side has exactly one extremum,
  // so the whole list is that one index.
  if (l0.count() == 0) l0 = MirrorList{0, 0, 0};
  if (l1.count() == 0) l1 = MirrorList{0, 0, 0};
  if (r0.count() == 0) r0 = MirrorList{nM - 1, nM - 1, 0};
  if (r1.count() == 0) r1 = MirrorList{nm - 1, nm - 1, 0};
  // sample index of entry j
  auto left_at = [&](const MirrorList& l, int q, int n, int j) {
    return l.hi - j >= l.lo ? ind_of(C, q, n, NB, l.hi - j) : 0;
  };
  auto right_at = [&](const MirrorList& l, int q, int n, int j) {
    if (l.end) return j == 0 ? N - 1 : ind_of(C, q, n, NB, l.lo + j - 1);
    return ind_of(C, q, n, NB, l.hi - j);
  };
  // ---- mirrored point does not reach the boundary (kernels.py:469-503) ----
  const real T0 = T(0), TN = T(N - 1);
  const real tl = T(lsym), tr = T(rsym);
  // the mirrored positions are stored as REAL_T before the compares
  // (kernels.py:471-472, 488-489): in the FP32 build that rounds them
  const real tl1 = 2.0 * tl - T(left_at(l1, 1, nm, 0)), tl0 = 2.0 * tl - T(left_at(l0, 0, nM, 0));
  if (tl1 > T0 || tl0 > T0) {
    if (lsym == im0) l0 = MirrorList{min(nM, NB) - 1, 0, 0};
    else l1 = MirrorList{min(nm, NB) - 1, 0, 0};
    lsym = 0;
  }
  const real tr1 = 2.0 * tr - T(right_at(r1, 1, nm, r1.count() - 1));
  const real tr0 = 2.0 * tr - T(right_at(r0, 0, nM, r0.count() - 1));
  if (tr1 < TN || tr0 < TN) {
    if (rsym == imL) r0 = MirrorList{nM - 1, max(nM - NB, 0), 0};
    else r1 = MirrorList{nm - 1, max(nm - NB, 0), 0};
    rsym = N - 1;
  }
  const int c0 = l0.count(), c1 = l1.count(), c2 = r0.count(), c3 = r1.count();
  if (lane == 0) {
    C.lsym = lsym;
    C.rsym = rsym;
    C.kbase[0] = NB - c0;
    C.kbase[1] = NB - c1;
    C.kcnt[0] = c0 + nM + c2;
    C.kcnt[1] = c1 + nm + c3;
  }
  // eight lanes a list write its knots: left maxima, left minima, right ones
  const int q = lane >> 3, side = q & 1;
  const bool left = q < 2;
  const MirrorList l = left ? (side == 0 ? l0 : l1) : (side == 0 ? r0 : r1);
  const int n = side == 0 ? nM : nm, cnt = l.count();
  const real sym = T(left ? lsym : rsym);
  real2* xy = (side == 0 ? K.XY[0] : K.XY[1]) + (left ? NB - cnt : NB + n);
  bool bad = false;
#pragma unroll 1
  for (int j = lane & 7; j < cnt; j += 8) {
    const int idx = left ? left_at(l, side, n, j) : right_at(l, side, n, j);
    const real val = S[idx];
    const real pos = 2.0 * sym - T(idx);
    xy[j] = real2{pos, val};
    bad |= side == 0 ? (val < 0.0) : (val > 0.0);
  }
  return bad;
}

// ---------------------------------------------------------------------------
// Not-a-knot spline: reduced system + PCR + moments (kernels.py:607-697).
// ---------------------------------------------------------------------------
// position of a knot of a pair array
struct PairX {
  const real2* p;
  __device__ __forceinline__ real operator[](int i) const { return p[i].x; }
};
struct PairY {
  const real2* p;
  __device__ __forceinline__ real operator[](int i) const { return p[i].y; }
};

// Row r of a PCR buffer: byte offset of its (a, c) pair; its (b, d) pair
// follows kBD bytes on.
constexpr int kRow = (int)sizeof(real2), kBD = 8 * kRow;
__device__ __forceinline__ int row_at(int r) { return (r >> 3) * (2 * kBD) + (r & 7) * kRow; }
// Byte distance to the row `s` below / above a row that is number r & 7 of its block
__device__ __forceinline__ int row_below(int r, int s) {
  return s < 8 ? s * kRow + ((r & 7) < s ? kBD : 0) : 2 * s * kRow;
}
__device__ __forceinline__ int row_above(int r, int s) {
  return s < 8 ? s * kRow + ((r & 7) + s >= 8 ? kBD : 0) : 2 * s * kRow;
}
__device__ __forceinline__ real2& pair_at(char* p) { return *reinterpret_cast<real2*>(p); }
__device__ __forceinline__ const real2& pair_at(const char* p) {
  return *reinterpret_cast<const real2*>(p);
}

// The quotient with its range test: FP64 from the approximate reciprocal where
// that is exact.
__device__ __forceinline__ real div_any(real a, real b) {
#if EMDB_F32
  return a / b;
#else
  bool slow = false;
  const real q = div_nb(a, b, slow);
  return slow ? div_slow(a, b) : q;
#endif
}

// The PCR levels from stride s on, each quotient tested, rows of two systems
// in buffer `cur` (kernels.py:651-668, in the reference's operation order);
// the result ends up in buffer 1.  The whole CTA calls it, for the systems that
// the levels in solve_splines do not cover.
template <int NT>
__device__ __noinline__ void pcr_levels_any(char* b0, char* b1, int m0, int m1, int s, int cur) {
  const int tid = threadIdx.x, mt = m0 + m1, guard = row_at(mt);
#pragma unroll 1
  for (; s < max(m0, m1); s *= 2) {
    const char* src = cur ? b1 : b0;
    char* dst = cur ? b0 : b1;
#pragma unroll 1
    for (int r = tid; r < mt; r += NT) {
      const bool s0 = r < m0;
      const bool hl = (s0 && r >= s) || r >= m0 + s;
      const bool hr = r < m0 - s || (!s0 && r < mt - s);
      const char* own = src + row_at(r);
      const char* l = src + (hl ? row_at(r - s) : guard);
      const char* rr = src + (hr ? row_at(r + s) : guard);
      const real2 o = pair_at(own), p = pair_at(own + kBD);
      const real2 ol = pair_at(l), pl = pair_at(l + kBD);
      const real2 orr = pair_at(rr), pr = pair_at(rr + kBD);
      const real alpha = hl ? div_any(o.x, pl.x) : real(0);
      const real beta = hr ? div_any(o.y, pr.x) : real(0);
      char* to = dst + row_at(r);
      pair_at(to) = real2{-alpha * ol.x, -beta * orr.y};
      pair_at(to + kBD) = real2{p.x - alpha * ol.y - beta * orr.x,
                                p.y - alpha * pl.y - beta * pr.y};
    }
    cur ^= 1;
    __syncthreads();
  }
  if (cur == 0) {
#pragma unroll 1
    for (int r = tid; r < mt; r += NT) {
      const int at = row_at(r);
      pair_at(b1 + at + kBD) = pair_at(b0 + at + kBD);
    }
    __syncthreads();
  }
}

// The last PCR level of a system whose multipliers have died out (see
// solve_splines): the right-hand side after it, d.  The diagonal stays as it
// is.  A neighbour's term is formed only where it can
// reach the rounding of d: RN(d - x) = d for |x| below a quarter ulp, and the
// magnitude words bound |a d_l| against |d b_l| from both sides (each is at
// most 0.0861 below its logarithm).
__device__ __forceinline__ real pcr_last(const char* own, const char* l, const char* r, bool hl,
                                         bool hr) {
  constexpr int kFrac = sizeof(real) == 8 ? 20 : 23;
  constexpr int kGap = ((sizeof(real) == 8 ? 55 : 26) << kFrac) + (1 << kFrac) / 4;
  const real2 o = pair_at(own), pl = pair_at(l + kBD), pr = pair_at(r + kBD);
  real d = pair_at(own + kBD).y;
  const int dm = (int)mag(d);
  if (hl && dm - (int)mag(o.x) <= (int)mag(pl.y) - (int)mag(pl.x) + kGap)
    d -= o.x / pl.x * pl.y;
  if (hr && dm - (int)mag(o.y) <= (int)mag(pr.y) - (int)mag(pr.x) + kGap)
    d -= o.y / pr.x * pr.y;
  return d;
}

// Spline rows, parallel cyclic reduction and the moments of both envelopes
// (kernels.py:607-697), every row rounded as the reference rounds it.
//
// The reference halves the coupling until the stride passes the system,
// ceil(log2 m) levels.  The multipliers square from level to level (1/4, 1/14,
// 1/194, 2^-15, 2^-30, 2^-61 on equal spacing; at most 1/2, 1/7, 1/97, ... on
// any), so from some level on no row changes any more, and those levels are
// left out once that is certain.  With every multiplier of the fifth level
// (stride 16) at most e <= 2^-26:
//   * the sixth has multipliers a_k/b_l = -alpha_k alpha_l <= e^2 (1 + 2^-40)
//     and the diagonal's changes, alpha_k beta_l b_k <= e^4 b_k, are far below
//     its half ulp: b is final after the fifth level;
//   * when the magnitudes of all d are within 2^46 of each other, the sixth
//     level changes none of them by more than 2^-5 of itself, and from the
//     seventh on, with multipliers of at most e^4 (1 + 2^-40), |alpha d_l| <
//     2^-104 2^47 |d| is below the quarter ulp: d cannot change either.
// (All magnitudes normal and finite, which the vote checks too.)
// What is left after five levels is the sixth level's d, in which most terms
// round away too (pcr_last), and the division by the diagonal, fused.  One
// vote decides for both systems; systems for which it fails (and those of at
// most 32 rows) run every level.
// Bound by FP64 latency and instruction supply: per row and level two
// quotients (20 FP64 operations), 8 more and about 45 others, six 16-byte
// loads.  On 2048-sample seismic traces the row-levels fall from 4.25 to 3.0
// million per 24 traces, at 8192 samples from 16.4 to 9.7; no pass of those
// needed a seventh level.  B200, all levels with the former quotients / cut
// short, 16-byte rows / blocks of rows, no operand tests, votes without
// reductions, plain divisions where a lane has one: 16,384 x 2048 seismic 84.8 /
// 72.7 / 54.2 ms (the last with the other changes since), 256 x 8192 89.0 / 66.9
// / 50.8, 96 x 1501 1.75 / 1.60 / 1.15; envelopes alone, 4,096 x 2048: 0.53 / 0.38
// / 0.35 ms.
//
// Quotients without range checks or zero tests.  Suppose the spacings are
// positive, within [2^-100, 2^100) and within 2^24 of each other, and no
// right-hand side is -0.  The rows stay diagonally dominant
// (|a| + |c| <= b/2; rows without a left or right neighbour <= b), so b loses
// at most half a level and stays within 2^-5 and 2^6 of the spacings; each
// level squares the couplings relative to it, so the non-zero ones entering
// the fifth level are at least 2^-52 (2^-30)^16 2^-100 = 2^-632 (2^-52: the
// end rows' h1 - h0), and their quotients' last remainders at least 2^-870:
// nothing underflows.  A zero coupling gives the multiplier +0 where the
// division may give -0, and a row without a neighbour multiplies a row (0, 1,
// 0, 0) by its zero coupling instead of by +0; either changes no b, and no d
// except -0 - (-0), which cannot arise from right-hand sides other than -0.
// Each row checks its spacing -- on the integer axis to be in [1, kMaxIntSeg],
// else within 2^12 of the first one -- and one vote decides; the others take
// pcr_levels_any, and so do the levels past the fifth where the vote on those
// fails (its window for d is 2^23 either way of the middle row's).
// Returns (the same in every thread) whether the evaluation needs no test of
// spacings and moments: on the integer axis the condition on spacings above, on
// a given one spacings in [2^-100, 2^100) -- however far from each other, so an
// axis with a gap of any length keeps it -- and every moment zero or in [2^-700,
// 2^900).
// FP32: the same on the integer axis.  A coupling entering the fourth level is
// a spacing times eight multipliers h_k / (2 (h_k + h_k+1)), each at least a
// quarter, or a quarter of h_k / h_k+1 where spacings rise: with at most four
// rises of 2^16 and one end row's factor it is at least 2^-96, and the
// remainders are exact.  The fifth level divides where one is below 2^-80
// (extrema in pairs thousands of samples apart).  Every float moment is in
// div6's range.  On a given axis the FP32 build divides, tests its segment
// quotients, and gets true.  B200, 4,096 x 1500 float seismic: 10.2 ms,
// evaluation without tests 9.2, and the rows too 8.2.
template <int NT, bool kInt>
__device__ __forceinline__ bool solve_splines(const Knots& K, int kbase0, int kbase1, int kcnt0,
                                              int kcnt1, int tid, Ctl& C) {
  constexpr bool kDouble = sizeof(real) == 8;
  constexpr int kLast = 32;                     // stride of the fused level
  constexpr int kFrac = kDouble ? 20 : 23, kBias = kDouble ? 1023 : 127;   // of magnitude words
  const int m0 = kcnt0 >= 4 ? kcnt0 - 2 : 0;
  const int m1 = kcnt1 >= 4 ? kcnt1 - 2 : 0;
  const int mt = m0 + m1, mmax = max(m0, m1);
  const real2* xy0 = K.XY[0] + kbase0;
  const real2* xy1 = K.XY[1] + kbase1;
  const bool deep = mmax > kLast;
  // levels alternate buffers and have to end in buffer 1 (M goes to buffer 0):
  // five of them, or ceil(log2 mmax)
  int cur = deep || mmax < 2 ? 0 : 1 ^ (1 & (32 - __clz(mmax - 1)));
  const int guard = row_at(mt);
  if (tid < 2) {
    // the neighbour of rows that have none
    pair_at(K.rows(tid) + guard) = real2{real(0), real(0)};
    pair_at(K.rows(tid) + guard + kBD) = real2{real(1), real(0)};
  }
  // Rows (kernels.py:613-636): row k has the segments k and k+1 around it, and
  // each segment's slope serves two rows.  A lane forms one slope and takes
  // its left neighbour's from the lane below, so a warp's 32 segments give 31
  // rows and the next 32 start one back: one division a row instead of two.
  // The end rows have the same right-hand side up to the factor h/(h0+h1).
  const int z0 = m0 > 0 ? m0 + 1 : 0, zt = z0 + (m1 > 0 ? m1 + 1 : 0);
  const unsigned href = kInt ? 0u : mag(xy0[1].x - xy0[0].x) - (12u << kFrac);
  bool odd = false;
  bool far = false;           // given axis: a spacing that the evaluation's quotients don't take
#pragma unroll 1
  for (int zb = (tid >> 5) * 31; zb < zt; zb += (NT / 32) * 31) {
    const int z = zb + (tid & 31);
    const bool s0 = z < z0;
    const int g = s0 ? z : z - z0, m = s0 ? m0 : m1;          // segment g of a system of m rows
    real h = real(1), sl = real(0);
    if (z < zt) {
      const real2* xy = (s0 ? xy0 : xy1) + g;
      const real2 p0 = xy[0], p1 = xy[1];
      h = p1.x - p0.x;
      sl = (p1.y - p0.y) / h;
      if (kInt) odd |= !(h >= real(1) && h <= real(kMaxIntSeg));
      else if (kDouble) {
        odd |= !(h > real(0)) || mag(h) - href >= (24u << kFrac);
        far |= !(h > real(0)) || mag(h) - ((kBias - 100u) << kFrac) >= (200u << kFrac);
      }
    }
    const real hm = __shfl_up_sync(kFull, h, 1), sm = __shfl_up_sync(kFull, sl, 1);
    if (z < zt && (tid & 31) != 0 && g > 0) {
      const int k = g - 1, r = (s0 ? 0 : m0) + k;
      real a = hm, b = 2.0 * (hm + h), c = h, d = 6.0 * (sl - sm);
      if (k == 0 || k == m - 1) {
        const real dh = k == 0 ? h * d : hm * d;
        d = dh / (hm + h);
        a = k == 0 ? real(0) : hm - h;
        b = k == 0 ? hm + 2.0 * h : 2.0 * hm + h;
        c = k == 0 ? h - hm : real(0);
      }
      char* to = K.rows(cur) + row_at(r);
      pair_at(to) = real2{a, c};
      pair_at(to + kBD) = real2{b, d};
      if (kDouble || kInt) odd |= d == real(0) && signbit(d);
    }
  }
  if (!kInt && kDouble) odd |= href - ((kBias - 100u) << kFrac) >= (176u << kFrac);
  const bool plain = !__syncthreads_or(odd);
  odd = kInt ? !plain : far;
  EMDB_PH(&C, 2);
  bool fused = false;
  int s = 1;
  if (plain) {
#pragma unroll 1
    for (; s < min(mmax, kLast); s *= 2) {
      const int below = row_below(tid, s), above = row_above(tid, s);
      const char* src = K.rows(cur);
      char* dst = K.rows(cur ^ 1);
      // the level whose multipliers and right-hand sides are looked at
      const bool vote = 2 * s == kLast && deep;
      const unsigned dref =
          mag(pair_at(src + row_at(mt >> 1) + kBD).y) - (23u << kFrac);
      bool no = dref - (1u << kFrac) >= unsigned(2 * kBias - 50) << kFrac;
      int at = row_at(tid);
#pragma unroll 1
      for (int r = tid; r < mt; r += NT, at += NT * 2 * kRow) {
        const bool s0 = r < m0;
        const bool hl = (s0 && r >= s) || r >= m0 + s;
        const bool hr = r < m0 - s || (!s0 && r < mt - s);
        const char* own = src + at;
        const char* l = hl ? own - below : src + guard;
        const char* rr = hr ? own + above : src + guard;
        const real2 o = pair_at(own), p = pair_at(own + kBD);
        const real2 ol = pair_at(l), pl = pair_at(l + kBD);
        const real2 orr = pair_at(rr), pr = pair_at(rr + kBD);
        real alpha, beta;
        if (kDouble || kInt) {
          alpha = div_core(o.x, pl.x), beta = div_core(o.y, pr.x);
#if EMDB_F32
          if (s == 16 && (tiny(o.x) || tiny(o.y))) {
            alpha = div_slow(o.x, pl.x);
            beta = div_slow(o.y, pr.x);
          }
#endif
        } else {
          alpha = hl ? o.x / pl.x : real(0), beta = hr ? o.y / pr.x : real(0);
        }
        const real2 p2{p.x - alpha * ol.y - beta * orr.x, p.y - alpha * pl.y - beta * pr.y};
        pair_at(dst + at) = real2{-alpha * ol.x, -beta * orr.y};
        pair_at(dst + at + kBD) = p2;
        if (vote)
          no |= max(mag(alpha), mag(beta)) > (kBias - 26u) << kFrac ||
                mag(p2.y) - dref >= (46u << kFrac) || (!kDouble && mag(p2.x) < (1u << kFrac));
      }
      cur ^= 1;
      if (vote) fused = !__syncthreads_or(no);
      else __syncthreads();
    }
  }
  if (!fused && s < mmax) pcr_levels_any<NT>(K.rows(0), K.rows(1), m0, m1, s, cur);
  EMDB_PH(&C, 3);
  // diagonal solve
  {
    const char* src = K.rows(1);
    int at = row_at(tid);
#pragma unroll 1
    for (int r = tid; r < mt; r += NT, at += NT * 2 * kRow) {
      const bool s0 = r < m0;
      const char* own = src + at;
      const real2 p = pair_at(own + kBD);
      real d = p.y;
      if (fused) {
        const bool hl = (s0 && r >= kLast) || r >= m0 + kLast;
        const bool hr = r < m0 - kLast || (!s0 && r < mt - kLast);
        d = pcr_last(own, hl ? own - 2 * kLast * kRow : own, hr ? own + 2 * kLast * kRow : own,
                     hl, hr);
      }
      const real q = d / p.x;
      (s0 ? K.M[0] : K.M[1])[s0 ? r + 1 : r - m0 + 1] = q;
      if (kDouble) odd |= odd_moment(q);
    }
  }
  __syncthreads();
  // end moments from the first and last two (the reference forms the same
  // quotients d/b again)
  if (tid < 4) {
    const int q = tid >> 1;
    const int n = q == 0 ? kcnt0 : kcnt1;
    if (n >= 4) {
      const PairX x{q == 0 ? xy0 : xy1};
      real* M = q == 0 ? K.M[0] : K.M[1];
      const bool left = (tid & 1) == 0;
      const int i = left ? 0 : n - 3;
      const real ha = x[i + 1] - x[i], hb = x[i + 2] - x[i + 1];
      // M[0] = ((h0+h1) M[1] - h0 M[2]) / h1, M[n-1] the same from the other end
      const real ho = left ? ha : hb, hi = left ? hb : ha;
      const real m = ((ha + hb) * M[left ? 1 : n - 2] - ho * M[left ? 2 : n - 3]) / hi;
      M[left ? 0 : n - 1] = m;
      if (kDouble) odd |= odd_moment(m);
    }
  }
  const int any_odd = __syncthreads_or(odd);
  EMDB_PH(&C, 4);
  return !any_odd;
}

// One envelope's spline: knots, moments, knot count, mirrored-left and true knots.
struct SideView {
  const real2* xy;
  const real* M;
  int n;
  int nl, nt;
};

// Envelope value at t in knot segment lo (kernels.py:706-733).
__device__ __forceinline__ real eval_seg(const SideView& s, real t, int lo) {
  const PairX x{s.xy};
  const PairY y{s.xy};
  if (s.n == 2) {
    real slope = (y[1] - y[0]) / (x[1] - x[0]);
    return y[0] + slope * (t - x[0]);
  }
  if (s.n == 3) {
    real l0 = (t - x[1]) * (t - x[2]) / ((x[0] - x[1]) * (x[0] - x[2]));
    real l1 = (t - x[0]) * (t - x[2]) / ((x[1] - x[0]) * (x[1] - x[2]));
    real l2 = (t - x[0]) * (t - x[1]) / ((x[2] - x[0]) * (x[2] - x[1]));
    return y[0] * l0 + y[1] * l1 + y[2] * l2;
  }
  real x0 = x[lo], x1 = x[lo + 1];
  real y0 = y[lo], y1 = y[lo + 1];
  real M0 = s.M[lo], M1 = s.M[lo + 1];
  real h = x1 - x0;
  real A = (x1 - t) / h;
  real B = (t - x0) / h;
  return A * y0 + B * y1 + ((A * A * A - A) * M0 + (B * B * B - B) * M1) * (h * h) / 6.0;
}

// eval_seg for n >= 4 knots with the quotients formed without the division's
// slow-path branch, in the same operation order; sets `slow` for operands
// outside the exact range, and the caller then re-evaluates the sample with
// eval_seg.  (FP64: spacings in [2^-100, 2^100), see EnvEval; the numerators'
// quotients as in div_nb from one reciprocal.)
__device__ __forceinline__ real eval_seg_q(const real2* xy, const real* M, real t, int lo,
                                           bool& slow) {
  const real2 p0 = xy[lo], p1 = xy[lo + 1];
  const real M0 = M[lo], M1 = M[lo + 1];
  const real h = p1.x - p0.x;
#if EMDB_F32
  const real rh = real(1) / h;
  const real A = div_q(p1.x - t, h, rh, slow);
  const real B = div_q(t - p0.x, h, rh, slow);
#else
  const real a = p1.x - t, b = t - p0.x;
  const real y = recip(h);
  const real A = quot(a, h, y), B = quot(b, h, y);
  slow |= odd_range(a) || odd_range(b);
#endif
  const real num = ((A * A * A - A) * M0 + (B * B * B - B) * M1) * (h * h);
  return (A * p0.y + B * p1.y) + div6(num, slow);
}

// The reference's per-sample binary search (kernels.py:722-726).
__device__ __forceinline__ int search_seg(const SideView& s, real t) {
  int lo = 0, hi = s.n - 2;
#pragma unroll 1
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (s.xy[mid].x <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Both envelopes at t by search and division, out of line: the rare passes'
// evaluation (fewer than 4 knots, knot lists that are not strictly increasing,
// operands outside the quotients' range), one call site a loop.
__device__ __noinline__ real2 eval_any(const real2* xy0, const real* M0, int n0,
                                       const real2* xy1, const real* M1, int n1, real t) {
  const SideView s0{xy0, M0, n0, 0, 0}, s1{xy1, M1, n1, 0, 0};
  return real2{eval_seg(s0, t, n0 >= 4 ? search_seg(s0, t) : 0),
               eval_seg(s1, t, n1 >= 4 ? search_seg(s1, t) : 0)};
}

// 128-lane tree of the reference (kernels.py:794-804), on warp 0, for a value
// each thread has stored at red[q*128 + tid].  op 0: sum, 1: fmax, 2: fmin.
__device__ __forceinline__ real lane_tree(const real* red, int lane, int op) {
  real v0 = red[lane], v1 = red[lane + 32], v2 = red[lane + 64], v3 = red[lane + 96];
  real r;
  if (op == 0) r = (v0 + v2) + (v1 + v3);
  else if (op == 1) r = fmax(fmax(v0, v2), fmax(v1, v3));
  else r = fmin(fmin(v0, v2), fmin(v1, v3));
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    real o = __shfl_down_sync(kFull, r, s);
    if (op == 0) r = r + o;
    else if (op == 1) r = fmax(r, o);
    else r = fmin(r, o);
  }
  return r;
}

struct PassSums {
  real sq, dsq, osq, std_, omax, omin;
  bool bad;
  bool oor;
};

__device__ __forceinline__ void accumulate(PassSums& ps, real old, real nw) {
  real diff = nw - old;
  ps.sq += nw * nw;
  ps.dsq += diff * diff;
  ps.osq += old * old;
  real qd = diff / nw;
  ps.std_ += qd * qd;
  ps.omax = fmax(ps.omax, old);
  ps.omin = fmin(ps.omin, old);
}

// The wide instances' stop-test sums after the update (new values in imf[],
// old ones in oldv[], quotients (new-old)/new in qbuf[]): the reference's 128
// lanes, lane l adding samples l, l+128, ... in increasing order exactly as
// accumulate() does.  The six sums are independent chains, so the CTA's
// 128-thread groups take them apart -- 512 threads: Σnew² | Σdiff² |
// Σold², max, min | Σquotient²; 256 threads: the first two | the rest --
// and write the lanes' partials to red[128 * sum + l] for the trees.
template <int NT>
__device__ __forceinline__ void wide_lane_sums(real* red, const real* __restrict__ oldv,
                                               const real* imf, const real* __restrict__ qbuf,
                                               int N, int tid) {
  constexpr int NG = NT / kThreads;
  static_assert(NG == 2 || NG == 4, "wide instances have 256 or 512 threads");
  const int g = tid / kThreads, l = tid % kThreads;
  if (g == 0) {
    real s = 0.0, s2 = 0.0;
#pragma unroll kLaneUnroll
    for (int i = l; i < N; i += kThreads) {
      const real nw = imf[i];
      s += nw * nw;
      if (NG == 2) {
        const real diff = nw - oldv[i];
        s2 += diff * diff;
      }
    }
    red[l] = s;
    if (NG == 2) red[128 + l] = s2;
  } else if (NG == 4 && g == 1) {
    real s = 0.0;
#pragma unroll kLaneUnroll
    for (int i = l; i < N; i += kThreads) {
      const real diff = imf[i] - oldv[i];
      s += diff * diff;
    }
    red[128 + l] = s;
  } else if (g == NG / 2) {
    real s = 0.0, mx = -1e30, mn = 1e30, sq = 0.0;
#pragma unroll kLaneUnroll
    for (int i = l; i < N; i += kThreads) {
      const real old = oldv[i];
      s += old * old;
      mx = fmax(mx, old);
      mn = fmin(mn, old);
      if (NG == 2) {
        const real q = qbuf[i];
        sq += q * q;
      }
    }
    red[256 + l] = s;
    red[512 + l] = mx;
    red[640 + l] = mn;
    if (NG == 2) red[384 + l] = sq;
  } else if (NG == 4 && g == 3) {
    real s = 0.0;
#pragma unroll kLaneUnroll
    for (int i = l; i < N; i += kThreads) {
      const real q = qbuf[i];
      s += q * q;
    }
    red[384 + l] = s;
  }
}

// eval_seg for the time axis T = arange(N) on a strictly increasing knot list
// of n >= 4 knots, t inside segment lo: knot positions (true and mirrored) and
// sample times are integers, so A = (x1-t)/h and B = (t-x0)/h are quotients of
// integers 0 <= a <= h.  For those, q0 = RN(a*y) with y = RN(1/h) and one
// correction RN(q0 + (a - h*q0)*y) equal RN(a/h): checked exhaustively for
// every pair with h <= 65536 (2.1e9 pairs).
//
// No operand is tested.  With h <= kMaxIntSeg and every moment zero or in
// [2^-700, 2^900) (EnvEval): A is 0, 1 or in [1/h, 1 - 1/h], so A^3 - A is 0 or
// at least 2^-18 and at most 1/2, its product with a moment 0 or a normal
// number of at least 2^-718, the sum of two such products a multiple of 2^-771
// below 2^900, and h^2 in [1, 2^32]: num is 0 or in [2^-771, 2^932), inside
// div6's range.  (FP32: every float is; its quotients take both corrections.)
__device__ __forceinline__ real eval_seg_int(const real2* xy, const real* M, real t, int lo) {
  const real2 p0 = xy[lo], p1 = xy[lo + 1];
  const real M0 = M[lo], M1 = M[lo + 1];
  const real h = p1.x - p0.x;
  const real a = p1.x - t, b = t - p0.x;
  const real r = recip(h);
#if EMDB_F32
  const real A = quot(a, h, r), B = quot(b, h, r);
#else
  real A = a * r;
  A = fma(fma(-A, h, a), r, A);
  real B = b * r;
  B = fma(fma(-B, h, b), r, B);
#endif
  const real num = ((A * A * A - A) * M0 + (B * B * B - B) * M1) * (h * h);
  return (A * p0.y + B * p1.y) + div6(num);
}

// Both envelopes at sample i (kernels.py:706-733).
//
// O(1) segments: for a strictly increasing knot list (nbsym <= 2, no flat
// runs -- a plateau extremum sits at the run's midpoint, not at its flagged
// first sample) the reference's binary search returns (number of knots at
// or left of t) - 1, clamped to [0, n-2].  Otherwise run the search.  The
// true knots at or left of a sample come from the scan's ballot masks
// (global chunk prefix + popc).  Every left-mirrored knot lies at or left
// of T[lsym] and every right-mirrored one at or right of T[rsym], so only
// the chunks outside [lsym, rsym) compare them one by one; inside, with at
// least one mirrored knot at each end, no clamp is needed either.
//
// `hot`, one value for the pass: the segments are O(1) and the quotients need
// no test (solve_splines' answer), so that a chunk runs straight through; a
// pass with exact zeros or flat runs, nbsym > 2, fewer than four knots or
// operands of unusual magnitude searches and divides sample by sample.
//
// A sample takes 31 FP64 operations per envelope on the integer axis.  The loop
// over chunks is kept rolled and two chunks a trip are slower: the pass is
// bound by instruction supply and issue more than by FP64 latency.  Operand
// tests and cold paths in the loop, RN(1/h) from a table / as here: 8 x 30011
// 2.82 / 2.43 ms, 2,048 x 2048 from host memory 14.6 / 13.6, 16,384 x 2048 seismic
// 60.1 / 58.2.
template <bool kInt>
struct EnvEval {
  const SideView s0, s1;
  const bool hot;
  const int cL, cR;              // chunks that need no compare with mirrored knots
  const unsigned incl;
  __device__ __forceinline__ EnvEval(const SmemLayout& L, const SideView& a, const SideView& b,
                                     int NB, bool trig, bool plain, int lane)
      : s0(a), s1(b), hot(NB <= 2 && !trig && a.n >= 4 && b.n >= 4 && plain),
        cL((L.ctl->lsym + 31) >> 5), cR(L.ctl->rsym >> 5),
        incl(lane == 31 ? kFull : ((2u << lane) - 1u)) {}
  // chunk c, this lane's sample time t
  __device__ __forceinline__ void operator()(const SmemLayout& L, int c, real t, real& emax,
                                             real& emin) const {
    bool slow = !hot;
    if (hot) {
      const uint2 m = L.mm[c];
      const uint32_t pp = L.pp[c];
      int lo0 = min((int)(pp & 0xffffu) + __popc(m.x & incl), s0.nt);
      int lo1 = min((int)(pp >> 16) + __popc(m.y & incl), s1.nt);
      if (c < cL || c >= cR) {
        // mirrored knots at or left of t
        int k0 = -1, k1 = -1;
#pragma unroll 1
        for (int j = 0; j < s0.nl + s1.nl; ++j) {
          const bool f = j < s0.nl;
          const bool in = (f ? s0.xy[j].x : s1.xy[j - s0.nl].x) <= t;
          k0 += f && in;
          k1 += !f && in;
        }
        const int e0 = s0.nl + s0.nt, e1 = s1.nl + s1.nt;
#pragma unroll 1
        for (int j = 0; j < (s0.n - e0) + (s1.n - e1); ++j) {
          const bool f = j < s0.n - e0;
          const bool in = (f ? s0.xy[e0 + j].x : s1.xy[e1 + j - (s0.n - e0)].x) <= t;
          k0 += f && in;
          k1 += !f && in;
        }
        lo0 = min(max(lo0 + k0, 0), s0.n - 2);
        lo1 = min(max(lo1 + k1, 0), s1.n - 2);
      } else {
        lo0 += s0.nl - 1;
        lo1 += s1.nl - 1;
      }
      if (kInt) {
        emax = eval_seg_int(s0.xy, s0.M, t, lo0);
        emin = eval_seg_int(s1.xy, s1.M, t, lo1);
      } else {
        emax = eval_seg_q(s0.xy, s0.M, t, lo0, slow);
        emin = eval_seg_q(s1.xy, s1.M, t, lo1, slow);
      }
    }
    if (slow) {
      const real2 v = eval_any(s0.xy, s0.M, s0.n, s1.xy, s1.M, s1.n, t);
      emax = v.x;
      emin = v.y;
    }
  }
};

// One sift pass after the extrema scan of the current proto-IMF: knots,
// mirroring, both splines, then the fused envelope / mean / update / partial
// sums.  kPlace selects where the knots live: shared memory (the common case),
// split between shared memory and the per-CTA global slab, or the slab alone.
//
// NT > 128 (the wide instance, one long trace per CTA): every thread
// evaluates samples, but the stop-test sums keep the reference's 128 lanes,
// each adding its samples in order.  So the proto-IMF is always parked in
// `park_old` (global, per CTA) while warp 0 mirrors, the evaluation writes the
// update to imf[] and its quotient diff/new to `qbuf`, and the first 128
// threads then sum old / new / quotient per lane exactly as accumulate() does.
template <int NT, int kGroup, bool kInt>
__device__ __forceinline__ int sift_pass(const SmemLayout& L, char* slab, const ExtInfo& e,
                                              int N, int NB, const TimeAxis& T, int tid, int warp,
                                              int lane, int place = kPlaceSmem,
                                              real* park_old = nullptr, real* qbuf = nullptr) {
  constexpr bool kWide = NT > kThreads;
  // kGroup >= 0: one placement, fixed at compile time.  kGroup == kOnChip /
  // kOffChip: one instance for the on-chip (shared, borrow) or off-chip
  // (split, park, slab) placements, chosen by `place` at run time.
  const int kPlace = kGroup >= 0 ? kGroup
                   : kGroup == kOnChip ? ((place == kPlaceBorrow || place == kPlaceBorrow2)
                                              ? kPlaceBorrow : kPlaceSmem)
                   : kGroup == kOffChip ? (place == kPlaceSplit ? kPlaceSplit
                                           : place == kPlacePark ? kPlacePark : kPlaceSlab)
                                        : place;
  Ctl& C = *L.ctl;
  real* imf = L.imf;
  const int kc0 = e.n_max + 2 * NB + 2, kc1 = e.n_min + 2 * NB + 2;
  Knots K = kPlace == kPlaceSmem    ? place_knots(L.arena, kc0, kc1)
           : kPlace == kPlaceSplit  ? place_knots_split(L.arena, L.arena_bytes, slab, kc0, kc1)
           : kPlace == kPlaceBorrow ? (place == kPlaceBorrow2
                                          ? place_knots_borrow2(imf, L.arena, L.arena_bytes, slab, N, kc0, kc1)
                                          : place_knots_borrow(imf, L.arena, L.arena_bytes, slab, N, kc0, kc1))
           : kPlace == kPlaceBorrow2 ? place_knots_borrow2(imf, L.arena, L.arena_bytes, slab, N, kc0, kc1)
           : kPlace == kPlacePark   ? place_knots_park(imf, slab, N, kc0, kc1, L.red)
                                    : place_knots(slab, kc0, kc1);
  PassSums ps;
  EMDB_PH(&C, 9);
  bool bad = fill_true_knots<scan_slots<NT>()>(L, K, e, N, NB, T, warp, lane);
  bad = __syncthreads_or(bad);
  EMDB_PH(&C, 0);
  bool mbad = false;
  const bool lend = kPlace == kPlaceBorrow || kPlace == kPlaceBorrow2 || kPlace == kPlacePark;
  // the wide instances also park it for the stop-test lanes, which read the
  // old samples back after the update
  const bool parked = lend || (kWide && !bad);
  if (warp == 0) {
    mbad = mirror_both(L, K, e, N, NB, T, lane);
  } else if (kWide) {
    if (parked)
#pragma unroll 1
      for (int i = tid - 32; i < N; i += NT - 32) park_old[i] = imf[i];
  } else if (lend) {
    // park the proto-IMF while warp 0 mirrors; the PCR buffers overwrite it
    real* save = borrow_save(slab);
#pragma unroll 1
    for (int i = tid - 32; i < N; i += kThreads - 32) save[i] = imf[i];
  }
  ps.bad = __syncthreads_or(bad || mbad) != 0;
  EMDB_PH(&C, 1);
  const int kb0 = C.kbase[0], kb1 = C.kbase[1], kn0 = C.kcnt[0], kn1 = C.kcnt[1];
  const bool plain = solve_splines<NT, kInt>(K, kb0, kb1, kn0, kn1, tid, C);
  const real* oldv = !parked ? imf : kWide ? park_old : borrow_save(slab);
  // A pass with a maximum below zero or a minimum above it is never the last
  // one of its IMF, whatever the stop tests say (the reference forms their
  // sums first and then drops them, kernels.py:773-776), so their terms,
  // lane sums and trees are formed for the other passes only: 19 % of the
  // passes of 2048-sample seismic traces, 9-11 % at 4096-8192.  B200, before /
  // after: 256 x 8192 seismic 104.2 / 97.9 ms, 96 x 1501 2.09 / 1.84 ms.
  const bool sums = !ps.bad;

  const SideView sv0{K.XY[0] + kb0, K.M[0], kn0, NB - kb0, e.n_max};
  const SideView sv1{K.XY[1] + kb1, K.M[1], kn1, NB - kb1, e.n_min};

  ps.sq = ps.dsq = ps.osq = ps.std_ = 0.0;
  ps.omax = -1e30;
  ps.omin = 1e30;
  bool oor = false;
  const EnvEval<kInt> eval(L, sv0, sv1, NB, e.trig, plain, lane);
  // T is strictly increasing, so the knot spans cover every sample iff they
  // cover the first and the last one
  if (N > 0) {
    const real t0 = T(0), tN = T(N - 1);
    oor = (t0 < sv0.xy[0].x) || (tN > sv0.xy[sv0.n - 1].x) || (t0 < sv1.xy[0].x) ||
          (tN > sv1.xy[sv1.n - 1].x);
  }
  // one warp a chunk of 32 samples, every NT / 32-th chunk (thread tid has the
  // samples tid, tid + NT, ...); lanes past the end compute the last sample again
  real ti = (real)tid;
#pragma unroll 1
  for (int c = __shfl_sync(kFull, warp, 0); c << 5 < N; c += NT / 32) {
    const int i = (c << 5) + lane;
    const real t = kInt ? ti : T(min(i, N - 1));
    ti += (real)NT;
    const real old = oldv[min(i, N - 1)];
    real emax, emin;
    eval(L, c, t, emax, emin);
    const real mean = 0.5 * (emax + emin);
    const real nw = old - mean;
    if (i < N) {
      imf[i] = nw;
      if (sums) {
        // the wide instances sum per reference lane after the update
        if (kWide) qbuf[i] = (nw - old) / nw;
        else accumulate(ps, old, nw);
      }
    }
  }
  // per-lane partial sums, then the reference's 128-lane trees on warp 0
  real* red = kPlace == kPlaceSlab ? L.red : K.red;
  if constexpr (kWide) {
    __syncthreads();
    EMDB_PH(&C, 5);
    if (sums) wide_lane_sums<NT>(red, oldv, imf, qbuf, N, tid);
  } else if (sums) {
    red[tid] = ps.sq; red[128 + tid] = ps.dsq; red[256 + tid] = ps.osq;
    red[384 + tid] = ps.std_; red[512 + tid] = ps.omax; red[640 + tid] = ps.omin;
  }
  __syncthreads();
  EMDB_PH(&C, kWide ? 6 : 5);
  // the six trees spread over the warps (warp w: sum w; warps 0/1 also the
  // max / min tree); the next extrema scan's barrier publishes C.sums
  if (sums && (!kWide || warp < kWarps)) {
    const real a = lane_tree(red + 128 * warp, lane, 0);
    if (lane == 0) C.sums[warp] = a;
    if (warp < 2) {
      const real b = lane_tree(red + 128 * (4 + warp), lane, 1 + warp);
      if (lane == 0) C.sums[4 + warp] = b;
    }
  }
  return (ps.bad ? 1 : 0) | (oor ? 2 : 0);
}

}  // namespace

// ---------------------------------------------------------------------------
// The sift kernel.
// ---------------------------------------------------------------------------
// Chunk completion for the host-memory pipeline (emdb_run_host): after the
// barrier that follows every output write of trace b, thread 0 raises its
// chunk's row maximum to the trace's count of rows that may hold data (rows
// beyond it are zero) and counts the trace in the chunk's device counter; the CTA that
// completes the chunk publishes it with one store of 1 + the chunk's row
// maximum to the chunk's flag in mapped host memory, so the host can copy just
// those rows of that chunk back while the rest of the batch sifts.  The device
// fence before the count and the system fence before the flag order all the
// chunk's output writes (from every CTA that counted) before the flag.
__device__ __forceinline__ void mark_trace_done(const SiftParams& p, int b, int tid, int nim) {
  if (p.chunk_count == nullptr || tid != 0) return;
  const int c = b / p.chunk_traces;
  atomicMax(p.chunk_rows + c, (unsigned)max(nim, 0));
  __threadfence();
  const unsigned need = (unsigned)min(p.chunk_traces, p.chunk_span - c * p.chunk_traces);
  if (atomicAdd(p.chunk_count + c, 1u) + 1u == need) {
    const unsigned rows = atomicMax(p.chunk_rows + c, 0u);
    __threadfence_system();
    *reinterpret_cast<volatile unsigned*>(p.chunk_flag + c) = 1u + rows;
  }
}

// NT threads per CTA: 128 (the reference's lanes), or 512 for the wide
// instance that gives one long trace a whole SM.  kMinBlocks is the
// register-budget variant: the compiler fits the kernel into
// 65536 / (NT * kMinBlocks) registers so that many CTAs can be resident.
// kGImf (wide only): the proto-IMF in the global slab, for traces longer than
// shared memory holds.
// kTail: the build that takes part in tail migration -- a 128/256-thread
// instance that hands its last traces over, or the 512-thread instance that
// resumes them (p.resume).  The other builds carry none of its code.
template <int NT, int kMinBlocks, bool kInt, bool kGImf = false, bool kTail = false>
__global__ void __launch_bounds__(NT, kMinBlocks) emd_sift_kernel(SiftParams p) {
  constexpr bool kWide = NT > kThreads;
  static_assert(!kGImf || kWide, "the global proto-IMF is built for the wide instance");
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int NB = p.nbsym;
  const int MAXI = p.max_imfs;
  Ctl* Cs = reinterpret_cast<Ctl*>(smem);
  char* slab = p.slab + (size_t)blockIdx.x * p.slab_stride;
  // wide instance: the parked proto-IMF and the stop-test quotients (and the
  // proto-IMF itself for kGImf), past the knot slab in this CTA's stride
  real* park_old = kWide ? reinterpret_cast<real*>(slab + p.park_off) : nullptr;
  real* qbuf = kWide ? reinterpret_cast<real*>(slab + p.q_off) : nullptr;
  real* gimf = kGImf ? reinterpret_cast<real*>(slab + p.imf_off) : nullptr;

  // this launch may hand over its tail / resumes another launch's tail
  const bool migrate = kTail && NT != kWideThreads && p.cont_buf != nullptr;
  const bool resume = kTail && NT == kWideThreads && p.resume != 0;
  for (;;) {
    if (tid == 0) Cs->job = atomicAdd(resume ? p.cont_ticket : p.queue, 1);
    __syncthreads();
    const int job = Cs->job;
    // a resume launch takes the continuation records instead of the queue
    const ContHead* rec = nullptr;
    if (resume) {
      if (job >= p.cont_cap) break;
      if (!p.cont_valid[job]) {
        __syncthreads();          // every thread has read Cs->job before it is reused
        continue;
      }
      rec = reinterpret_cast<const ContHead*>(p.cont_buf + (size_t)job * p.cont_stride);
    } else if (job >= p.batch) {
      break;
    }
    const int b = rec ? rec->b : p.order ? p.order[job] : job;
    const int64_t off = p.offsets ? p.offsets[b] : (int64_t)b * p.dense_n;
    const int N = p.offsets ? (int)(p.offsets[b + 1] - off) : p.dense_n;
    const real* S = p.values + off;
    real* out = p.imfs + (int64_t)MAXI * off;
    TimeAxis T;
    T.arange = kInt;            // the launch picks the build by p.t_mode
    T.T = p.t_mode == kTShared ? p.T : (p.t_mode == kTPerTrace ? p.T + off : nullptr);

    if (fixed_bytes<NT, kGImf>(N) + kRedBytes + 64 > (size_t)p.arena_bytes ||
        (kWide && p.q_off + (size_t)N * sizeof(real) > p.slab_stride) ||
        (kGImf && p.imf_off + (size_t)N * sizeof(real) > p.slab_stride)) {
      // cannot hold this trace: report, leave outputs flagged
      if (tid == 0) {
        atomicOr(p.status, kStatusTooLong);
        p.n_imfs[b] = 0;
        p.overflow[b] = 1;
        if (migrate) atomicAdd(p.started, 1);   // the others wait for all to have started
      }
      for (int k = tid; k < MAXI; k += NT) {
        p.dbg_n[(int64_t)b * MAXI + k] = -1;
        p.dbg_ext[(int64_t)b * MAXI + k] = -1;
        p.dbg_nzm[(int64_t)b * MAXI + k] = -1;
      }
      __syncthreads();
      mark_trace_done(p, b, tid, MAXI);     // rows unwritten: the host copies them all
      continue;
    }
    SmemLayout L = carve<NT, kGImf>(smem, N, p.arena_bytes, gimf);
    Ctl& C = *L.ctl;
    real* imf = L.imf;
    if (migrate && tid == 0) {
      atomicAdd(p.active, 1);
      atomicAdd(p.started, 1);
    }
    for (int k = tid; k < MAXI; k += NT) {
      C.dbg_n[k] = rec ? rec->dbg[0][k] : -1;
      C.dbg_e[k] = rec ? rec->dbg[1][k] : -1;
      C.dbg_z[k] = rec ? rec->dbg[2][k] : -1;
    }
#if EMDB_LOAD_CLOCKS
    const long long clk_trace0 = clock64();
#endif
    {
      // a resumed trace restarts from its parked proto-IMF
      const real* src = rec ? reinterpret_cast<const real*>(reinterpret_cast<const char*>(rec) +
                                                          cont_data_off())
                            : S;
      for (int i = tid; i < N; i += NT) imf[i] = src[i];
    }
    __syncthreads();
#if EMDB_LOAD_CLOCKS
    if (tid == 0 && p.counters)
      atomicAdd(p.counters + 2, (unsigned long long)(clock64() - clk_trace0));
    if (tid == 0) {
      for (int k = 0; k < kPhases; ++k) C.ph[k] = 0;
      C.ph_last = clock64();
    }
#endif

    bool ovf = rec ? rec->ovf != 0 : false;
    int imf_count = rec ? rec->imf_count : 0;
    bool finished = false;
    int extNo_last = rec ? rec->extNo_last : -1;
    bool stale = rec ? rec->stale != 0 : false;
    const int n_resume = rec ? rec->n : 0;
    bool yielded = false;
    int n_yield = 0;
    unsigned long long passes = 0, spilled = 0;

    // One loop over scans: each sift pass and each emitted IMF row ends in an
    // extrema scan of the proto-IMF it leaves, which is also the next pass's
    // (the reference scans the same data twice, kernels.py:930 vs 965).  One
    // copy of the scan, the pass and the emission keeps the loop small.
    int n = n_resume;
    bool post = false;          // the scan follows a sift pass
    bool pass_bad = false;
    for (;;) {
      const ExtInfo e = extrema_scan<NT>(L, N, tid, warp, lane, p.max_extrema);
      EMDB_PH(&C, 7);
      ovf |= e.overflow;
      const int extNo = e.n_max + e.n_min;
      bool emit = false;
      if (post) {
        extNo_last = extNo;
        if (!pass_bad && abs(extNo - e.n_zer) < 2) {
          const real sum_new_sq = C.sums[0], diff_sq = C.sums[1], old_sq = C.sums[2];
          const real std_sum = C.sums[3], omax = C.sums[4], omin = C.sums[5];
          bool f1 = false;
          if (sum_new_sq < kSumNewSqMin) f1 = false;
          else if (diff_sq / (omax - omin) < kSvarThr) f1 = true;
          else if (std_sum < kStdThr) f1 = true;
          else if (diff_sq / old_sq < kEnergyRatioThr) f1 = true;
          if (f1) {
            if (tid == 0) { C.dbg_n[imf_count] = n; C.dbg_e[imf_count] = extNo; C.dbg_z[imf_count] = e.n_zer; }
            emit = true;
          }
        }
      }
      if (!emit) {
        if (migrate && (n & 3) == 0) {
          // every trace has started and few remain: hand this one to the
          // 512-thread instance at this pass boundary (checked every fourth
          // pass: the two L2 reads and the barrier cost ~1 % per pass).  A record
          // holds the longest trace the launch was announced (max_n); a longer
          // one that fits the arena all the same finishes here
          int want = 0;
          if (tid == 0)
            want = *reinterpret_cast<volatile int*>(p.started) >= p.total &&
                   *reinterpret_cast<volatile int*>(p.active) <= p.yield_below &&
                   cont_data_off() + (size_t)N * sizeof(real) <= p.cont_stride;
          if (__syncthreads_or(want)) {
            yielded = true;
            n_yield = n;
            break;
          }
        }
        ++n;
        if (n >= p.max_iteration) {
          ovf = true;
          if (tid == 0) { C.dbg_n[imf_count] = n; C.dbg_e[imf_count] = -1; C.dbg_z[imf_count] = -1; }
          emit = true;
        } else if (!(extNo > 2 && e.n_max >= 1 && e.n_min >= 1)) {
          extNo_last = extNo;
          finished = true;
          emit = true;
        }
      }
      if (emit) {
        // ---- emit IMF row, running residue into the next row and imf[], end
        // condition ----
        EMDB_PH(&C, 9);
        const real* rsrc = imf_count == 0 ? S : out + (int64_t)imf_count * N;
        real* row = out + (int64_t)imf_count * N;
        real* rnext = out + (int64_t)(imf_count + 1) * N;
        real gmax = -1e30, gmin = 1e30, gabs = 0.0;
        auto note = [&](real rn) {
          gmax = fmax(gmax, rn);
          gmin = fmin(gmin, rn);
          gabs += fabs(rn);
        };
        // four samples' residues in flight (the rows may alias as far as the
        // compiler knows, so it does not hoist loads over stores itself)
        for (int i0 = tid; i0 < N; i0 += 4 * NT) {
          real r[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) r[q] = rsrc[min(i0 + q * NT, N - 1)];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + q * NT;
            if (i < N) {
              const real v = imf[i];
              const real rn = r[q] - v;
              row[i] = v;
              rnext[i] = rn;
              imf[i] = rn;
              if (!kWide) note(rn);
            }
          }
        }
        if (kWide) {
          // the reference's 128 lanes
          __syncthreads();
          if (tid < kThreads)
            for (int i = tid; i < N; i += kThreads) note(imf[i]);
        }
        real* red = L.red;
        if (!kWide || tid < kThreads) { red[tid] = gmax; red[128 + tid] = gmin; red[256 + tid] = gabs; }
        __syncthreads();
        if (warp == 0) {
          real a0 = lane_tree(red, lane, 1);
          real a1 = lane_tree(red + 128, lane, 2);
          real a2 = lane_tree(red + 256, lane, 0);
          if (lane == 0) { C.sums[6] = a0 - a1; C.sums[7] = a2; }
        }
        __syncthreads();
        ++imf_count;
        if (C.sums[6] < kRangeThr || C.sums[7] < kTotalPowerThr) finished = true;
        EMDB_PH(&C, 8);
        if (finished || imf_count >= MAXI - 1) break;
        n = 0;
        post = false;
        continue;
      }
      // the wide instance's stride also holds the parked proto-IMF and the
      // quotients: its knots may use only the part before them
      const int kc0 = e.n_max + 2 * NB + 2, kc1 = e.n_min + 2 * NB + 2;
      const int place = choose_place(N, L.arena_bytes, kWide ? p.park_off : p.slab_stride,
                                     kc0, kc1, kGImf);
      int flags;
      if (place == kPlaceSmem || place == kPlaceBorrow || place == kPlaceBorrow2)
        flags = sift_pass<NT, kOnChip, kInt>(L, slab, e, N, NB, T, tid, warp, lane, place,
                                             park_old, qbuf);
      else
        flags = sift_pass<NT, kOffChip, kInt>(L, slab, e, N, NB, T, tid, warp, lane, place,
                                              park_old, qbuf);
      spilled += place != kPlaceSmem;
      ++passes;
      pass_bad = (flags & 1) != 0;
      stale |= (flags & 2) != 0;
      post = true;
    }

    if (yielded) {
      // continuation record in this CTA's slot (a CTA hands over at most one
      // trace: the queue is empty when it does)
      const int rec_id = p.cont_base + blockIdx.x;
      ContHead* h = reinterpret_cast<ContHead*>(p.cont_buf + (size_t)rec_id * p.cont_stride);
      real* dst = reinterpret_cast<real*>(reinterpret_cast<char*>(h) + cont_data_off());
      for (int i = tid; i < N; i += NT) dst[i] = imf[i];
      for (int k = tid; k < kMaxImfsCap; k += NT) {
        h->dbg[0][k] = C.dbg_n[k];
        h->dbg[1][k] = C.dbg_e[k];
        h->dbg[2][k] = C.dbg_z[k];
      }
      if (tid == 0) {
        h->b = p.trace0 + b;
        h->n = n_yield;
        h->imf_count = imf_count;
        h->extNo_last = extNo_last;
        h->ovf = ovf ? 1 : 0;
        h->stale = stale ? 1 : 0;
        p.cont_valid[rec_id] = 1;
        atomicSub(p.active, 1);
        if (p.counters) {
          atomicAdd(p.counters, passes);
          atomicAdd(p.counters + 1, spilled);
        }
      }
      __syncthreads();
      continue;
    }

    // ---- epilogue: trend removal, residue ~ 0 test, zero unused rows ----
    const int last_row = imf_count;   // row holding the running residue (or none if 0 IMFs)
    const bool trend = extNo_last <= 2 && imf_count > 0;
    if (trend) imf_count -= 1;
    const real* rres = last_row == 0 ? S : out + (int64_t)last_row * N;
    // the last proto-IMF (imf[] holds the residue): the row before the residue's
    const real* vlast = out + (int64_t)max(last_row - 1, 0) * N;
    real amax = 0.0;
    for (int i = tid; i < (!kWide || tid < kThreads ? N : 0); i += kThreads) {
      real r = rres[i];
      if (trend) r = r + vlast[i];
      amax = fmax(amax, fabs(r));
    }
    real* red = L.red;
    if (!kWide || tid < kThreads) red[tid] = amax;
    __syncthreads();
    if (warp == 0) {
      real a = lane_tree(red, lane, 1);
      if (lane == 0) C.sums[0] = a;
    }
    __syncthreads();
    const bool rzero = C.sums[0] <= kResidueZeroAtol;
    const int nim = rzero ? imf_count : imf_count + 1;
    for (int i = tid; i < N; i += NT) {
      if (trend) {
        real r = rres[i] + vlast[i];
        if (!rzero) out[(int64_t)imf_count * N + i] = r;
        out[(int64_t)last_row * N + i] = 0.0;
      } else {
        if (rzero && last_row < MAXI) out[(int64_t)last_row * N + i] = 0.0;
        else if (last_row == 0) out[i] = S[i];
      }
    }
    const int first_zero = last_row + 1;
    for (int64_t k = (int64_t)first_zero * N + tid; k < (int64_t)MAXI * N; k += NT) out[k] = 0.0;
    if (tid == 0) {
      p.n_imfs[b] = nim;
      p.overflow[b] = ovf ? 1 : 0;
      if (p.counters) {
        atomicAdd(p.counters, passes);
        atomicAdd(p.counters + 1, spilled);
      }
      if (migrate) atomicSub(p.active, 1);
    }
    if (stale) atomicOr(p.status, kStatusStaleEnvelope);
    for (int k = tid; k < MAXI; k += NT) {
      p.dbg_n[(int64_t)b * MAXI + k] = C.dbg_n[k];
      p.dbg_ext[(int64_t)b * MAXI + k] = C.dbg_e[k];
      p.dbg_nzm[(int64_t)b * MAXI + k] = C.dbg_z[k];
    }
    __syncthreads();
#if EMDB_LOAD_CLOCKS
    if (tid == 0 && p.counters) {
      atomicAdd(p.counters + 3, (unsigned long long)(clock64() - clk_trace0));
      for (int k = 0; k < kPhases; ++k) atomicAdd(p.counters + 4 + k, C.ph[k]);
    }
#endif
    // rows that may hold data: n_imfs, plus the dropped trend row that a
    // ~zero residue leaves in place (as the reference does)
    mark_trace_done(p, b, tid, nim + ((trend && rzero) ? 1 : 0));
  }
}

// ---------------------------------------------------------------------------
// Envelope-only diagnostic (envelope_batch_kernel, kernels.py:1100-1166):
// extrema + mirroring + both envelopes on raw traces, no sift loop.  The
// reference scans with find_extrema_serial here; the extrema lists are the
// same as the sift scan's (plateau rule included) and n_zer is not reported.
// ---------------------------------------------------------------------------
// kInt: integer time axis (T = arange), with the sift's evaluation; any other
// axis, which this entry point takes as it is given, is searched per sample.
template <bool kSmem, bool kInt>
__device__ __forceinline__ void envelope_pass(const SmemLayout& L, char* slab, const ExtInfo& e,
                                              int N, int NB, const TimeAxis& T, int tid, int warp,
                                              int lane, real* emax_out, real* emin_out,
                                              real* kp[2], real* kv[2], int mbuf, int nk[2],
                                              int* status) {
  Ctl& C = *L.ctl;
  const int kc0 = e.n_max + 2 * NB + 2, kc1 = e.n_min + 2 * NB + 2;
  Knots K = place_knots(kSmem ? L.arena : slab, kc0, kc1);
  fill_true_knots<kWarps>(L, K, e, N, NB, T, warp, lane);
  __syncthreads();
  if (warp == 0) mirror_both(L, K, e, N, NB, T, lane);
  __syncthreads();
  const int kb0 = C.kbase[0], kb1 = C.kbase[1], kn0 = C.kcnt[0], kn1 = C.kcnt[1];
  const bool plain = solve_splines<kThreads, kInt>(K, kb0, kb1, kn0, kn1, tid, C);
  const SideView sv[2] = {{K.XY[0] + kb0, K.M[0], kn0, NB - kb0, e.n_max},
                          {K.XY[1] + kb1, K.M[1], kn1, NB - kb1, e.n_min}};
  nk[0] = kn0;
  nk[1] = kn1;
  const int kcnt[2] = {kn0, kn1};
  bool oor = false;
  const EnvEval<kInt> eval(L, sv[0], sv[1], NB, e.trig, plain, lane);
#pragma unroll 1
  for (int ch = __shfl_sync(kFull, warp, 0); ch << 5 < N; ch += kWarps) {
    const int i = (ch << 5) + lane;
    const real t = T(min(i, N - 1));
    if (kInt) {
      // arange: the knot span covers every sample (see the mirroring)
      real a, b;
      eval(L, ch, t, a, b);
      if (i < N) {
        emax_out[i] = a;
        emin_out[i] = b;
      }
      continue;
    }
    if (i >= N) continue;
    int lo0 = sv[0].n >= 4 ? search_seg(sv[0], t) : 0;
    int lo1 = sv[1].n >= 4 ? search_seg(sv[1], t) : 0;
    bool r0 = !(t < sv[0].xy[0].x || t > sv[0].xy[sv[0].n - 1].x);
    bool r1 = !(t < sv[1].xy[0].x || t > sv[1].xy[sv[1].n - 1].x);
    real a = eval_seg(sv[0], t, lo0);
    real c = eval_seg(sv[1], t, lo1);
    emax_out[i] = r0 ? a : 0.0;
    emin_out[i] = r1 ? c : 0.0;
    oor |= !(r0 && r1);
  }
  if (oor) atomicOr(status, kStatusStaleEnvelope);
  for (int q = 0; q < 2; ++q)
    for (int k = tid; k < mbuf; k += kThreads) {
      kp[q][k] = k < kcnt[q] ? sv[q].xy[k].x : 0.0;
      kv[q][k] = k < kcnt[q] ? sv[q].xy[k].y : 0.0;
    }
}

template <bool kInt>
__global__ void __launch_bounds__(kThreads, 4) emd_envelope_kernel(EnvParams p) {
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int NB = p.nbsym;
  Ctl* Cs = reinterpret_cast<Ctl*>(smem);
  char* slab = p.slab + (size_t)blockIdx.x * p.slab_stride;
  for (;;) {
    if (tid == 0) Cs->job = atomicAdd(p.queue, 1);
    __syncthreads();
    const int b = Cs->job;
    if (b >= p.batch) break;
    const int64_t off = p.offsets ? p.offsets[b] : (int64_t)b * p.dense_n;
    const int N = p.offsets ? (int)(p.offsets[b + 1] - off) : p.dense_n;
    const real* S = p.values + off;
    real* emax_out = p.max_env + off;
    real* emin_out = p.min_env + off;
    real* kp[2] = {p.max_kpos + (int64_t)b * p.mbuf, p.min_kpos + (int64_t)b * p.mbuf};
    real* kv[2] = {p.max_kval + (int64_t)b * p.mbuf, p.min_kval + (int64_t)b * p.mbuf};
    TimeAxis T;
    T.arange = kInt;
    T.T = p.t_mode == kTShared ? p.T : (p.t_mode == kTPerTrace ? p.T + off : nullptr);
    if (fixed_bytes(N) + kRedBytes + 64 > (size_t)p.arena_bytes) {
      if (tid == 0) {
        atomicOr(p.status, kStatusTooLong);
        p.degenerate[b] = 1;
        p.n_extrema[2 * b] = 0; p.n_extrema[2 * b + 1] = 0;
        p.n_mirrored[2 * b] = 0; p.n_mirrored[2 * b + 1] = 0;
      }
      __syncthreads();
      continue;
    }
    SmemLayout L = carve<kThreads>(smem, N, p.arena_bytes);
    for (int i = tid; i < N; i += kThreads) L.imf[i] = S[i];
    __syncthreads();
    ExtInfo e = extrema_scan<kThreads>(L, N, tid, warp, lane, p.max_extrema);
    const bool degenerate = !(e.n_max + e.n_min > 2 && e.n_max >= 1 && e.n_min >= 1);
    int nk[2] = {0, 0};
    if (!degenerate) {
      const int kc0 = e.n_max + 2 * NB + 2, kc1 = e.n_min + 2 * NB + 2;
      if (knot_bytes(kc0, kc1) <= (size_t)L.arena_bytes)
        envelope_pass<true, kInt>(L, slab, e, N, NB, T, tid, warp, lane, emax_out, emin_out, kp, kv,
                            p.mbuf, nk, p.status);
      else
        envelope_pass<false, kInt>(L, slab, e, N, NB, T, tid, warp, lane, emax_out, emin_out, kp, kv,
                             p.mbuf, nk, p.status);
    } else {
      for (int i = tid; i < N; i += kThreads) { emax_out[i] = 0.0; emin_out[i] = 0.0; }
      for (int q = 0; q < 2; ++q)
        for (int k = tid; k < p.mbuf; k += kThreads) { kp[q][k] = 0.0; kv[q][k] = 0.0; }
    }
    if (tid == 0) {
      p.degenerate[b] = degenerate ? 1 : 0;
      p.n_extrema[2 * b] = e.n_max;
      p.n_extrema[2 * b + 1] = e.n_min;
      p.n_mirrored[2 * b] = nk[0];
      p.n_mirrored[2 * b + 1] = nk[1];
    }
    __syncthreads();
  }
}

#if !EMDB_F32
// ---------------------------------------------------------------------------
// Self-test of div_rn against the hardware division.  mode 0: every integer
// pair 0 <= a <= b <= n (the operands of A and B on the default time axis,
// where knot spacings are integers <= 2N); mode 1: n pseudo-random pairs with
// significands and exponents spread over [2^-600, 2^600] plus numerators
// formed like the spline's h^2-scaled term over 6.  Modes 2 and 3: the forms
// without a reciprocal at hand, see there.  Counts mismatching bits.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__global__ void div_check_kernel(int mode, long long n, unsigned long long seed,
                                 unsigned long long* mismatches) {
  unsigned long long bad0 = 0, bad1 = 0, bad2 = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (mode == 0) {
    // pairs indexed by b in [1, n]: thread grid-strides over b, loops over a
    for (long long bb = 1 + blockIdx.x * (long long)blockDim.x + threadIdx.x; bb <= n; bb += stride) {
      const double b = (double)bb;
      const double y = 1.0 / b;
      if (recip(b) != y) ++bad1;
      for (long long aa = 0; aa <= bb; ++aa) {
        const double a = (double)aa;
        if (__double_as_longlong(div_rn(a, b, y)) != __double_as_longlong(a / b)) ++bad0;
      }
    }
  } else if (mode == 2) {
    // div_nb: [0] random a/b over [2^-1100, 2^1100] (zeros, subnormals, infinities
    // through the fallback), [1] all-ones / power-of-two significands of b,
    // [2] PCR-like |a| <= |b| within 2^+-40 of 1
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
      uint64_t h1 = mix64(seed ^ (uint64_t)i), h2 = mix64(h1 ^ 0x5bd1e995ull);
      double ma = __longlong_as_double((long long)((h1 >> 12) | 0x3ff0000000000000ull));
      double mb = __longlong_as_double((long long)((h2 >> 12) | 0x3ff0000000000000ull));
      double a = ldexp(ma, (int)(h1 % 2201) - 1100), b = ldexp(mb, (int)(h2 % 2201) - 1100);
      if (h1 & 1) a = -a;
      if (h2 & 2) b = -b;
      bool slow = false;
      double q = div_nb(a, b, slow);
      if (slow) q = div_slow(a, b);
      if (__double_as_longlong(q) != __double_as_longlong(div_slow(a, b))) ++bad0;
      const int eb2 = (int)((h2 >> 20) % 161) - 80;
      double b2 = (h2 & 4) ? ldexp(__longlong_as_double(0x3fffffffffffffffll), eb2) : ldexp(1.0, eb2);
      if (h2 & 8) b2 = -b2;
      slow = false;
      q = div_nb(a, b2, slow);
      if (slow) q = div_slow(a, b2);
      if (__double_as_longlong(q) != __double_as_longlong(div_slow(a, b2))) ++bad1;
      double b3 = ldexp(mb, (int)((h2 >> 30) % 81) - 40);
      double a3 = b3 * ((double)((h1 >> 11) & 0xfffffffffffffull) * 0x1p-52);
      if (h1 & 16) a3 = -a3;
      slow = false;
      q = div_nb(a3, b3, slow);
      if (slow) q = div_slow(a3, b3);
      if (__double_as_longlong(q) != __double_as_longlong(div_slow(a3, b3))) ++bad2;
    }
  } else if (mode == 3) {
    // the quotients as the kernels use them, without a fallback.  PCR rows:
    // div_core for couplings from 2^-632 up and diagonals of spacings in [2^-100,
    // 2^100) (solve_splines), [0] random, [1] the smallest couplings over all-ones,
    // nearly all-ones and power-of-two significands; [2] segment quotients of
    // a given axis: quot with recip, 0 <= a <= h, a from 2^-900 (eval_seg_q)
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
      const uint64_t h1 = mix64(seed ^ (uint64_t)i), h2 = mix64(h1 ^ 0x5bd1e995ull);
      const uint64_t h3 = mix64(h2 ^ 0x9e3779b9ull);
      const double ma = __longlong_as_double((long long)((h1 >> 12) | 0x3ff0000000000000ull));
      const double mb = __longlong_as_double((long long)((h2 >> 12) | 0x3ff0000000000000ull));
      const int eb = (int)(h3 % 211) - 105;
      double a = ldexp(ma, -632 + (int)((h3 >> 8) % (unsigned)(eb + 634)));
      if (h1 & 1) a = -a;
      double b = ldexp(mb, eb);
      if (__double_as_longlong(div_core(a, b)) != __double_as_longlong(div_slow(a, b))) ++bad0;
      a = ldexp(ma, -632 + (int)((h3 >> 28) % 121));
      b = (h2 & 4) ? __longlong_as_double(0x3fffffffffffffffll - (long long)((h2 >> 3) & 15)) : 1.0;
      b = ldexp(b, eb);
      if (h2 & 2) a = -a;
      if (__double_as_longlong(div_core(a, b)) != __double_as_longlong(div_slow(a, b))) ++bad1;
      const int eh = (int)((h3 >> 40) % 200) - 100;
      const double h = ldexp(mb, eh);
      a = (h1 & 2) ? h * ((double)((h1 >> 11) & 0xfffffffffffffull) * 0x1p-52)
                   : ldexp(ma, -900 + (int)((h3 >> 48) % (unsigned)(eh + 900)));
      if (__double_as_longlong(quot(a, h, recip(h))) != __double_as_longlong(div_slow(a, h))) ++bad2;
    }
  } else {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
      uint64_t h1 = mix64(seed ^ (uint64_t)i), h2 = mix64(h1 ^ 0x5bd1e995ull);
      // significands in [1,2), exponents in [-300, 300] (quotients stay in range), random signs
      double ma = __longlong_as_double((long long)((h1 >> 12) | 0x3ff0000000000000ull));
      double mb = __longlong_as_double((long long)((h2 >> 12) | 0x3ff0000000000000ull));
      int ea = (int)(h1 % 601) - 300, eb = (int)(h2 % 601) - 300;
      double a = ldexp(ma, ea), b = ldexp(mb, eb);
      if (h1 & 1) a = -a;
      if (h2 & 2) b = -b;
      if (__double_as_longlong(div_rn(a, b, 1.0 / b)) != __double_as_longlong(a / b)) ++bad0;
      // division by 6 (the spline term's divisor)
      bool slow = false;
      double q6 = div6(a, slow);
      if (slow) q6 = div_slow(a, 6.0);
      if (__double_as_longlong(q6) != __double_as_longlong(a / 6.0)) ++bad1;
      // segment quotients: 0 <= a <= b, b a spacing in [1, 65536] with a random fraction
      double bi = (double)((h2 >> 40) % 65536 + 1) + (double)((h2 >> 8) & 0xffff) * 0x1p-16;
      double ai = bi * ((double)((h1 >> 11) & 0xfffffffffffffull) * 0x1p-52);
      if (__double_as_longlong(div_rn(ai, bi, 1.0 / bi)) != __double_as_longlong(ai / bi)) ++bad2;
    }
  }
  if (bad0) atomicAdd(mismatches, bad0);
  if (bad1) atomicAdd(mismatches + 1, bad1);
  if (bad2) atomicAdd(mismatches + 2, bad2);
}

cudaError_t launch_div_check(int mode, long long n, unsigned long long seed,
                             unsigned long long* mismatches, cudaStream_t stream) {
  div_check_kernel<<<148 * 8, 256, 0, stream>>>(mode, n, seed, mismatches);
  return cudaGetLastError();
}
#endif

#if EMDB_F32
// ---------------------------------------------------------------------------
// Self-test of the float quotients above against the float division.  mode 0:
// every integer pair 0 <= a <= b <= n through [0] div_q with y = RN(1/b) and [1]
// quot with recip(b); [2] div_core, every numerator over the 64 significands
// nearest 2.  mode 1: n pseudo-random pairs, [0] div_q with y = RN(1/b),
// significands random and exponents in [-40, 40]; [1] div_core (the division for
// `tiny` numerators) with exponents from -110 and of b in [-5, 23]; [2] div_core
// on PCR-like rows, |a| <= |b|; mode 2: div_core alone, [0] numerators from 2^-102,
// [1] the smallest over special significands, [2] every numerator of 2^-96 over
// the 64 significands nearest 2.  Counts mismatching bits.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64f(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ float rnd_float(uint64_t h, int e_lo, int e_hi) {
  const float m = __int_as_float((int)((h >> 41) | 0x3f800000u));     // [1, 2)
  const float v = ldexpf(m, (int)(h % (uint64_t)(e_hi - e_lo + 1)) + e_lo);
  return (h & (1ull << 20)) ? -v : v;
}

__global__ void div_check_f32_kernel(int mode, long long n, unsigned long long seed,
                                     unsigned long long* mismatches) {
  unsigned long long bad0 = 0, bad1 = 0, bad2 = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  auto wrong = [](float q, float a, float b) {
    return __float_as_int(q) != __float_as_int(div_slow(a, b));
  };
  if (mode == 0) {
    for (long long bb = 1 + first; bb <= n; bb += stride) {
      const float b = (float)bb;
      const float y = 1.0f / b, r = recip(b);
      for (long long aa = 0; aa <= bb; ++aa) {
        const float a = (float)aa;
        bool slow = false;
        float q = div_q(a, b, y, slow);
        if (slow) q = div_slow(a, b);
        bad0 += wrong(q, a, b);
        bad1 += wrong(quot(a, b, r), a, b);
      }
    }
    for (long long i = first; i < 64ll << 23; i += stride) {
      const float b = __int_as_float(0x3fffffff - (int)(i >> 23));             // 2 - (k + 1) 2^-23
      const float a = __int_as_float(0x3f800000 | (int)(i & 0x7fffff));
      bad2 += wrong(div_core(a, b), a, b);
    }
  } else if (mode == 2) {
    // div_core as the PCR rows use it, without a fallback: couplings from 2^-102
    for (long long i = first; i < n; i += stride) {
      const uint64_t h1 = mix64f(seed ^ (uint64_t)i), h2 = mix64f(h1 ^ 0x5bd1e995ull);
      const uint64_t h3 = mix64f(h2 ^ 0x9e3779b9ull);
      float a = rnd_float(h1, -102, 23), b = rnd_float(h2, -5, 23);
      bad0 += wrong(div_core(a, b), a, b);
      a = rnd_float(h3, -102, -80);
      b = (h1 & 2) ? __int_as_float(0x3fffffff - (int)((h2 >> 3) & 63)) : 1.0f;
      b = ldexpf(b, (int)((h3 >> 32) % 29) - 5);
      bad1 += wrong(div_core(a, b), a, b);
    }
    for (long long i = first; i < 64ll << 23; i += stride) {
      const float b = __int_as_float(0x3fffffff - (int)(i >> 23)) * 0x1p+22f;
      const float a = __int_as_float(0x3f800000 | (int)(i & 0x7fffff)) * 0x1p-96f;
      bad2 += wrong(div_core(a, b), a, b);
    }
  } else {
    for (long long i = first; i < n; i += stride) {
      const uint64_t h1 = mix64f(seed ^ (uint64_t)i), h2 = mix64f(h1 ^ 0x5bd1e995ull);
      const uint64_t h3 = mix64f(h2 ^ 0x9e3779b9ull), h4 = mix64f(h3 ^ 0x7f4a7c15ull);
      {
        const float a = rnd_float(h1, -40, 40), b = rnd_float(h2, -40, 40);
        bool slow = false;
        float q = div_q(a, b, 1.0f / b, slow);
        if (slow) q = div_slow(a, b);
        bad0 += wrong(q, a, b);
      }
      {
        const float a = rnd_float(h3, -110, 23), b = rnd_float(h4, -5, 23);
        bad1 += wrong(tiny(a) ? div_slow(a, b) : div_core(a, b), a, b);
      }
      {
        const float b = rnd_float(h2 ^ h3, -5, 23);
        const float f = __int_as_float((int)((h4 >> 41) | 0x3f800000u)) - 1.0f;   // [0, 1)
        const float a = ((h1 & 2) ? -f : f) * b;
        bad2 += a != 0.0f && wrong(div_core(a, b), a, b);
      }
    }
  }
  if (bad0) atomicAdd(mismatches, bad0);
  if (bad1) atomicAdd(mismatches + 1, bad1);
  if (bad2) atomicAdd(mismatches + 2, bad2);
}

cudaError_t launch_div_check(int mode, long long n, unsigned long long seed,
                             unsigned long long* mismatches, cudaStream_t stream) {
  div_check_f32_kernel<<<148 * 8, 256, 0, stream>>>(mode, n, seed, mismatches);
  return cudaGetLastError();
}
#endif

size_t sift_fixed_smem(int N, int variant, bool imf_global) {
  const int nt = variant_threads(variant);
  if (nt <= kThreads) return fixed_bytes(N) + kRedBytes;
  if (nt == kHalfWideThreads) return fixed_bytes<kHalfWideThreads>(N) + kRedBytes;
  return (imf_global ? fixed_bytes<kWideThreads, true>(N) : fixed_bytes<kWideThreads>(N)) +
         kRedBytes;
}

int sift_pass_placement(int N, int arena_total, size_t slab_stride, int kc0, int kc1) {
  const size_t fixed = fixed_bytes(std::max(N, 1));
  if (arena_total < 0 || (size_t)arena_total < fixed + kRedBytes + 64) return -1;
  return choose_place(N, arena_total - (int)fixed, slab_stride, kc0, kc1);
}

size_t sift_slab_bytes(int max_extrema, int nbsym) {
  const long long kc = (long long)max_extrema + 2LL * nbsym + 2;
  const size_t cap = (size_t)(2 * kc);
  const size_t red_extra = (4 * cap >= (size_t)kRedDoubles) ? 0 : kRedBytes;
  return align16(10 * cap * sizeof(real) + red_extra);
}

namespace {
// kInt: the kernel build for the integer time axis (T = arange), whose
// segment quotients are quotients of integers.
template <int NT, int V, bool kInt, bool kG = false>
cudaError_t occupancy_vt(int arena_bytes, int* ctas_per_sm) {
  cudaError_t e = cudaFuncSetAttribute(emd_sift_kernel<NT, V, kInt, kG>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, arena_bytes);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm,
                                                       emd_sift_kernel<NT, V, kInt, kG>, NT,
                                                       arena_bytes);
}
// CTAs per SM that both builds reach (the smaller), so a plan's grid fits either
template <int NT, int V, bool kG = false>
cudaError_t occupancy_v(int arena_bytes, int* ctas_per_sm) {
  int a = 0, b = 0;
  cudaError_t e = occupancy_vt<NT, V, true, kG>(arena_bytes, &a);
  if (e == cudaSuccess) e = occupancy_vt<NT, V, false, kG>(arena_bytes, &b);
  *ctas_per_sm = a < b ? a : b;
  return e;
}
template <int NT, int V, bool kInt, bool kG = false, bool kT = false>
cudaError_t launch_vt(const SiftParams& p, int grid, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(emd_sift_kernel<NT, V, kInt, kG, kT>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, p.arena_bytes);
  if (e != cudaSuccess) return e;
  emd_sift_kernel<NT, V, kInt, kG, kT><<<grid, NT, p.arena_bytes, stream>>>(p);
  return cudaGetLastError();
}
template <int NT, int V, bool kG = false, bool kT = false>
cudaError_t launch_v(const SiftParams& p, int grid, cudaStream_t stream) {
  return p.t_mode == kTArange ? launch_vt<NT, V, true, kG, kT>(p, grid, stream)
                              : launch_vt<NT, V, false, kG, kT>(p, grid, stream);
}
}  // namespace

#if !EMDB_F32
bool sift_variant_ok(int v) { return v == 1 || v == 2 || v == 4 || v == 5 || v == 6; }

int variant_threads(int v) {
  return v == 1 ? kWideThreads : v == 2 ? kHalfWideThreads : kThreads;
}
#endif

cudaError_t sift_occupancy(int arena_bytes, int variant, int* ctas_per_sm, bool imf_global) {
  switch (variant) {
    case 1: return imf_global ? occupancy_v<kWideThreads, 1, true>(arena_bytes, ctas_per_sm)
                              : occupancy_v<kWideThreads, 1>(arena_bytes, ctas_per_sm);
    case 2: return occupancy_v<kHalfWideThreads, 2>(arena_bytes, ctas_per_sm);
    case 5: return occupancy_v<kThreads, 5>(arena_bytes, ctas_per_sm);
    case 6: return occupancy_v<kThreads, 6>(arena_bytes, ctas_per_sm);
    default: return occupancy_v<kThreads, 4>(arena_bytes, ctas_per_sm);
  }
}

cudaError_t launch_sift(const SiftParams& p, int grid, cudaStream_t stream) {
  // tail migration (p.cont_buf): the 128 x 4 (FP32: and x 5) and 256 x 2 builds that hand over,
  // the 512-thread build that resumes
  if (p.cont_buf != nullptr) {
    switch (p.variant) {
      case 1: return launch_v<kWideThreads, 1, false, true>(p, grid, stream);
      case 4: return launch_v<kThreads, 4, false, true>(p, grid, stream);
#if EMDB_F32
      case 5: return launch_v<kThreads, 5, false, true>(p, grid, stream);
#endif
      case 2: return launch_v<kHalfWideThreads, 2, false, true>(p, grid, stream);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (p.variant) {
    case 1: return p.imf_off ? launch_v<kWideThreads, 1, true>(p, grid, stream)
                             : launch_v<kWideThreads, 1>(p, grid, stream);
    case 2: return launch_v<kHalfWideThreads, 2>(p, grid, stream);
    case 5: return launch_v<kThreads, 5>(p, grid, stream);
    case 6: return launch_v<kThreads, 6>(p, grid, stream);
    default: return launch_v<kThreads, 4>(p, grid, stream);
  }
}

namespace {
template <bool kInt>
cudaError_t envelope_occupancy_t(int arena_bytes, int* ctas_per_sm) {
  cudaError_t e = cudaFuncSetAttribute(emd_envelope_kernel<kInt>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, arena_bytes);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, emd_envelope_kernel<kInt>,
                                                       kThreads, arena_bytes);
}
template <bool kInt>
cudaError_t launch_envelope_t(const EnvParams& p, int grid, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(emd_envelope_kernel<kInt>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, p.arena_bytes);
  if (e != cudaSuccess) return e;
  emd_envelope_kernel<kInt><<<grid, kThreads, p.arena_bytes, stream>>>(p);
  return cudaGetLastError();
}
}  // namespace

// CTAs per SM that both builds reach
cudaError_t envelope_occupancy(int arena_bytes, int* ctas_per_sm) {
  int a = 0, b = 0;
  cudaError_t e = envelope_occupancy_t<true>(arena_bytes, &a);
  if (e == cudaSuccess) e = envelope_occupancy_t<false>(arena_bytes, &b);
  *ctas_per_sm = a < b ? a : b;
  return e;
}

cudaError_t launch_envelope(const EnvParams& p, int grid, cudaStream_t stream) {
  return p.t_mode == kTArange ? launch_envelope_t<true>(p, grid, stream)
                              : launch_envelope_t<false>(p, grid, stream);
}

}  // namespace emdb
