// fixsum.cuh -- sums of doubles on the integer pipe.
//
// GB300 retires one FP64 warp instruction per 64 clocks and SM sub-partition
// (1.9 FMA per clock per SM), and a butterfly sum of one double per lane takes
// 810 clocks (five dependent shuffle + DADD, ~120 clocks each, measured on one
// warp).  A warp reduction of a 32-bit integer (redux.sync) takes 45.  The
// sums here are therefore formed in fixed point: each addend p is placed in a
// 96-bit window below a bound 2^E (|p| < 2^E, by Cauchy-Schwarz from the norms
// of the vectors that are dotted, where they are known), cut into four signed
// 24-bit pieces, and the pieces are summed as integers: over a warp by
// four redux.sync, over a block and over the grid as two 64-bit limbs.
//
// The window holds every addend above 2^(E-43) exactly and cuts the others at
// 2^(E-96), so the sum is exact to 2^(E-96) per addend, whatever their number
// and order, which lets the blocks of a grid add into one pair of words with
// atomics instead of publishing partials that every block has to read back and
// add up.  That is more accurate than FP64 additions while the sum's largest
// addends are near the bound, and less where all of them are far below it: the
// callers look at how far.  An addend outside the window (Inf, NaN, or a bound
// that does not hold) is reported by the return value, and the sum is not taken.
#pragma once

#include "common.cuh"

namespace psf {

constexpr long long kFixMask48 = (1ll << 48) - 1;

// The four signed 24-bit pieces of p 2^(96-E), lowest first; false (pieces
// meaningless) when |p| >= 2^E or p is not finite.
PSF_DEVINL bool fix96_pieces(double p, int E, int (&b)[4]) {
  const unsigned hi = (unsigned)__double2hiint(p), lo = (unsigned)__double2loint(p);
  const int ex = (int)((hi >> 20) & 0x7ffu);
  const int pos = max(ex, 1) - (E + 979);  // p = m 2^(ex - 1075), the window's unit 2^(E - 96)
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (ex ? 0x100000u : 0u)) << 32) | lo;
  m >>= min(max(-pos, 0), 63);
  const int ls = min(max(pos, 0), 43);
  const unsigned long long l = m << ls;
  const unsigned h0 = (unsigned)(m >> (48 - ls));
  const unsigned h1 = (unsigned)((m >> (48 - ls)) >> 24);
  const int s = (int)hi >> 31;
  b[0] = ((int)((unsigned)l & 0xffffffu) ^ s) - s;
  b[1] = ((int)((unsigned)(l >> 24) & 0xffffffu) ^ s) - s;
  b[2] = ((int)(h0 & 0xffffffu) ^ s) - s;
  b[3] = ((int)h1 ^ s) - s;
  return pos <= 43 && ex != 0x7ff;
}

// Warp sum of the pieces (32 x 24 bits fit an int) as two limbs.
PSF_DEVINL void fix96_warp(const int (&b)[4], long long& hi, long long& lo) {
  const int s0 = __reduce_add_sync(0xffffffffu, b[0]), s1 = __reduce_add_sync(0xffffffffu, b[1]);
  const int s2 = __reduce_add_sync(0xffffffffu, b[2]), s3 = __reduce_add_sync(0xffffffffu, b[3]);
  lo = (long long)s0 + ((long long)s1 << 24);
  hi = (long long)s2 + ((long long)s3 << 24);
}

// lo into [0, 2^48), its carry into hi.
PSF_DEVINL void fix96_carry(long long& hi, long long& lo) {
  hi += lo >> 48;
  lo &= kFixMask48;
}

// (hi 2^48 + lo) 2^(E-96) as a double (one rounding of the sum; |hi| < 2^53).
PSF_DEVINL double fix96_value(long long hi, long long lo, int E) {
  fix96_carry(hi, lo);
  return scale_pow2(fma((double)hi, 281474976710656.0, (double)lo), E - 96);
}

PSF_DEVINL void red_add_s64(long long* p, long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// A word that other blocks add to inside this launch (read past L1).
PSF_DEVINL long long ld_relaxed_s64(const long long* p) {
  long long v;
  asm volatile("ld.relaxed.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// A still wider window for a squared norm that may be rounding noise of its
// bound: p 2^(192-E) as four 48-bit limbs, lowest first; p >= 0.
PSF_DEVINL bool fix192_limbs(double p, int E, long long (&w)[4]) {
  const unsigned hi = (unsigned)__double2hiint(p), lo = (unsigned)__double2loint(p);
  const int ex = (int)((hi >> 20) & 0x7ffu);
  int pos = max(ex, 1) - (E + 883);  // p = m 2^(ex - 1075), the window's unit 2^(E - 192)
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (ex ? 0x100000u : 0u)) << 32) | lo;
  const bool ok = pos <= 139 && ex != 0x7ff && (hi >> 31) == 0u;
  m >>= min(max(-pos, 0), 63);
  pos = min(max(pos, 0), 139);
  const int q = pos >= 96 ? 2 : pos >= 48 ? 1 : 0;  // the limb that holds the lowest bit
  const int ls = pos - 48 * q;
  const long long l = (long long)((m << ls) & (unsigned long long)kFixMask48), h = (long long)(m >> (48 - ls));
  w[0] = q == 0 ? l : 0;
  w[1] = q == 0 ? h : q == 1 ? l : 0;
  w[2] = q == 1 ? h : q == 2 ? l : 0;
  w[3] = q == 2 ? h : 0;
  return ok;
}

// The value of N 48-bit limbs, lowest first, in units of their window.
template <int N>
PSF_DEVINL double fix_units(long long (&w)[N]) {
#pragma unroll
  for (int q = 0; q + 1 < N; ++q) fix96_carry(w[q + 1], w[q]);
  double v = (double)w[N - 1];
#pragma unroll
  for (int q = N - 2; q >= 0; --q) v = fma(v, 281474976710656.0, (double)w[q]);  // 2^48
  return v;
}

// A non-zero addend with a mantissa bit below a window's unit 2^U.
PSF_DEVINL bool fix_cut(double p, int U) {
  const unsigned hi = (unsigned)__double2hiint(p) & 0x7fffffffu;
  return (hi | (unsigned)__double2loint(p)) != 0u && max((int)(hi >> 20), 1) - 1075 < U;
}
// |p| < 2^E (Inf and NaN are not).
PSF_DEVINL bool fix_below(double p, int E) { return (int)((__double2hiint(p) >> 20) & 0x7ff) - 1022 <= min(E, 1024); }

// ---------------------------------------------------------------------------
// Grid sums whose words count their own arrivals.  Each block adds to every
// limb's word, beside its signed 48-bit limb, 1 in the bits from 56 up; a
// reader that finds G there has the sum.  The arrival and the value are one
// word, so a reduction over the grid is one atomic and one L2 round trip past
// the last block, where a counter barrier, the fetch of every block's partial
// and their FP64 butterfly took 5500-6500 clocks (152 blocks; polling one slot
// per block instead of one word per limb is no cure: 152 x 152 polls made the
// same reduction 3000 clocks slower).  G <= 200.  The words start at
// count_start, whose bias keeps the sums of the limbs positive, so that the
// arrivals are the top byte as it is.
//
// The window is placed by a bound that the sum may stay far below (or, where
// the bound does not hold, lie above), so the sum itself says whether it
// stands.  The top word has, above a 40-bit limb, two more 8-bit counts: of
// the blocks whose addend has bits below the window's unit (bits 40-47), and
// of those whose addend is not below 2^(E-17) (bits 48-55; the others' top
// limbs are at most 2^31, and 200 of them below 2^39).  Each cut addend is off
// by less than one unit, so a total of 2^62 units or more is off by less than
// 2^-54 of itself, and one without cut addends is exact.  Otherwise the reader
// has to sum in FP64.
// ---------------------------------------------------------------------------
constexpr int kCountMaxBlocks = 200;
constexpr long long kCountOne = 1ll << 56;
constexpr long long kCountBad = 1ll << 48;
constexpr long long kCountCut = 1ll << 40;
constexpr int kCountHeadBits = 17;  // of the top limb's 48, above an addend
constexpr long long kCountLowBias = 1ll << 55, kCountTopBias = 1ll << 39;

// What word q of N starts at.
__host__ __device__ constexpr long long count_start(int q, int N) {
  return q + 1 < N ? kCountLowBias : kCountTopBias;
}

// ok: the addend is below 2^(E-17); cut: it has bits below the unit.
template <int N>
PSF_DEVINL void count_post(long long* words, long long (&w)[N], bool ok, bool cut) {
#pragma unroll
  for (int q = 0; q + 1 < N; ++q) {  // limbs into [-2^47, 2^47)
    const long long carry = (w[q] + (1ll << 47)) >> 48;
    w[q] -= carry << 48;
    w[q + 1] += carry;
  }
  const long long flag = cut ? kCountOne + kCountCut : kCountOne;
#pragma unroll
  for (int q = 0; q + 1 < N; ++q) red_add_s64(words + q, w[q] + kCountOne);
  red_add_s64(words + N - 1, ok ? w[N - 1] + flag : kCountOne + kCountBad);
}

// One thread: waits (bounded) for G arrivals on each word; the sum in units of
// the window, and whether it stands.
template <int N>
PSF_DEVINL bool count_wait(const long long* words, int G, double& units, bool& stands, int* err) {
  long long w[N];
  unsigned long long t0 = 0;
  for (unsigned n = 0;; ++n) {
    bool all = true;
#pragma unroll
    for (int q = 0; q < N; ++q) w[q] = ld_relaxed_s64(words + q);
#pragma unroll
    for (int q = 0; q < N; ++q) all &= (int)((unsigned long long)w[q] >> 56) == G;
    if (all) break;
    if ((n & 63u) == 63u) {
      if (t0 == 0) t0 = globaltimer_ns();
      if (*(volatile int*)err != 0) return false;
      if (globaltimer_ns() - t0 > kWaitLimitNs) {
        atomicOr(err, DEVERR_TIMEOUT);
        return false;
      }
    }
  }
  const unsigned flags = (unsigned)((unsigned long long)w[N - 1] >> 40) & 0xffffu;
#pragma unroll
  for (int q = 0; q + 1 < N; ++q) w[q] = (w[q] & (kCountOne - 1)) - kCountLowBias;
  w[N - 1] = (w[N - 1] & (kCountCut - 1)) - kCountTopBias;
  units = fix_units(w);
  stands = flags == 0u;
  if (!stands) stands = flags < 0x100u && fabs(units) >= 4611686018427387904.0;  // no bad addend, 2^62
  return true;
}

// The same sum in FP64, by one warp of every block: the partials of all blocks
// in `part`, their arrivals counted in *arrivals (zero before), the total (a
// fixed order) in *out, in shared memory.  False when the wait gave up.
static __device__ __noinline__ bool count_sum_fp64(double mine, double* part, long long* arrivals, int bid, int G,
                                                   int* err, double* out) {
  const int lane = threadIdx.x & 31;
  int ok = 1;
  if (lane == 0) {
    *(volatile double*)(part + bid) = mine;
    __threadfence();
    red_add_s64(arrivals, 1);
    const unsigned long long t0 = globaltimer_ns();
    while (ld_relaxed_s64(arrivals) < G) {
      if (*(volatile int*)err != 0) { ok = 0; break; }
      if (globaltimer_ns() - t0 > kWaitLimitNs) {
        atomicOr(err, DEVERR_TIMEOUT);
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
    __threadfence();
  }
  __syncwarp();
  ok = __shfl_sync(0xffffffffu, ok, 0);
  double v = 0.0;
  if (ok)
    for (int b = lane; b < G; b += 32) v += *(const volatile double*)(part + b);
  v = warp_sum(v);
  if (lane == 0) *out = v;
  return ok != 0;
}

}  // namespace psf
