// fixsum.cuh -- sums of doubles on the integer pipe.
//
// GB300 retires one FP64 warp instruction per 64 clocks and SM sub-partition
// (1.9 FMA per clock per SM), and a butterfly sum of one double per lane takes
// 810 clocks (five dependent shuffle + DADD, ~120 clocks each, measured on one
// warp).  A warp reduction of a 32-bit integer (redux.sync) takes 45.  The
// sums here are therefore formed in fixed point: each addend p is placed in a
// 96-bit window below a bound 2^E known beforehand (|p| < 2^E, by
// Cauchy-Schwarz from the norms of the vectors that are dotted), cut into four
// signed 24-bit pieces, and the pieces are summed as integers: over a warp by
// four redux.sync, over a block and over the grid as two 64-bit limbs.
//
// The window holds every addend above 2^(E-43) exactly and cuts the others at
// 2^(E-96), so the sum is exact to 2^(E-96) per addend, whatever their number:
// more accurate than any FP64 order of additions, and the same bits for every
// order, which lets the blocks of a grid add into one pair of words with
// atomics instead of publishing partials that every block has to read back and
// add up.  An addend outside the window (Inf, NaN, or a bound that does not
// hold) is reported by the return value; the callers turn the sum into NaN.
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

// A wider window for sums that may be far below their bound (the squared norm
// of what Gram-Schmidt leaves): p 2^(144-E) as three 48-bit limbs, lowest
// first, exact for p >= 2^(E-91); p >= 0.
PSF_DEVINL bool fix144_limbs(double p, int E, long long (&w)[3]) {
  const unsigned hi = (unsigned)__double2hiint(p), lo = (unsigned)__double2loint(p);
  const int ex = (int)((hi >> 20) & 0x7ffu);
  int pos = max(ex, 1) - (E + 931);
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (ex ? 0x100000u : 0u)) << 32) | lo;
  const bool ok = pos <= 91 && ex != 0x7ff && (hi >> 31) == 0u;
  const bool top = pos >= 48;
  if (top) pos -= 48;
  m >>= min(max(-pos, 0), 63);
  const int ls = min(max(pos, 0), 47);
  const long long l = (long long)((m << ls) & (unsigned long long)kFixMask48), h = (long long)(m >> (48 - ls));
  w[0] = top ? 0 : l;
  w[1] = top ? l : h;
  w[2] = top ? h : 0;
  return ok;
}

PSF_DEVINL double fix144_value(long long w2, long long w1, long long w0, int E) {
  w1 += w0 >> 48;
  w0 &= kFixMask48;
  w2 += w1 >> 48;
  w1 &= kFixMask48;
  const double c = 281474976710656.0;  // 2^48
  return scale_pow2(fma(fma((double)w2, c, (double)w1), c, (double)w0), E - 144);
}

PSF_DEVINL long long warp_sum_s64(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
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

PSF_DEVINL double fix192_value(long long w3, long long w2, long long w1, long long w0, int E) {
  w1 += w0 >> 48;
  w0 &= kFixMask48;
  w2 += w1 >> 48;
  w1 &= kFixMask48;
  w3 += w2 >> 48;
  w2 &= kFixMask48;
  const double c = 281474976710656.0;  // 2^48
  const double v = fma(fma(fma((double)w3, c, (double)w2), c, (double)w1), c, (double)w0);
  return scale_pow2(v, E - 192);
}

// ---------------------------------------------------------------------------
// Grid sums whose words count their own arrivals.  Each block adds to every
// limb's word, beside its signed 48-bit limb, 1 in the bits from 56 up; a
// reader that finds G there has the sum.  The arrival and the value are one
// word, so a reduction over the grid is one atomic and one L2 round trip past
// the last block, where a counter barrier, the fetch of every block's partial
// and their FP64 butterfly took 5500-6500 clocks (152 blocks; polling one slot
// per block instead of one word per limb is no cure: 152 x 152 polls made the
// same reduction 3000 clocks slower).  G <= 200; a block whose addend does not
// fit the window marks the top limb, and the sum becomes NaN: the bound E
// passed to it lies 3 bits above what the sum can reach, which keeps unmarked
// top limbs below 2^46.
// ---------------------------------------------------------------------------
constexpr int kCountMaxBlocks = 200;
constexpr long long kCountOne = 1ll << 56;
constexpr long long kCountMark = 1ll << 47;

template <int N>
PSF_DEVINL void count_post(long long* words, long long (&w)[N], bool ok) {
#pragma unroll
  for (int q = 0; q + 1 < N; ++q) {  // limbs into [-2^47, 2^47)
    const long long carry = (w[q] + (1ll << 47)) >> 48;
    w[q] -= carry << 48;
    w[q + 1] += carry;
  }
  if (!ok) w[N - 1] = kCountMark;
#pragma unroll
  for (int q = 0; q < N; ++q) red_add_s64(words + q, w[q] + kCountOne);
}

// One thread: waits (bounded) for G arrivals on each word; w the sums.
template <int N>
PSF_DEVINL bool count_wait(const long long* words, int G, long long (&w)[N], bool& ok, int* err) {
  unsigned long long t0 = 0;
  for (unsigned n = 0;; ++n) {
    bool all = true;
#pragma unroll
    for (int q = 0; q < N; ++q) w[q] = ld_relaxed_s64(words + q);
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const long long c = (long long)((unsigned long long)(w[q] + (1ll << 55)) >> 56);
      all &= c == G;
      w[q] -= (long long)((unsigned long long)c << 56);
    }
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
  ok = w[N - 1] < (1ll << 46) && w[N - 1] > -(1ll << 46);
  return true;
}

}  // namespace psf
