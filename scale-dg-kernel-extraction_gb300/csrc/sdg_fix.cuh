// 60-bit fixed-point arithmetic for the FP64 line sums.
//
// GB300 issues a 32 x 32 + 64 bit integer multiply-add (IMAD.WIDE) 36 times
// as fast as an FP64 FMA (58-61 against 1.66 a clock and SM, measured), so a
// product of two 60-bit numbers, formed from a 31-bit and a 29-bit limb by
// three of them, costs a twelfth of a DFMA.  The values of one line share a power-of-two
// scale; sums of products are then exact integer sums, independent of their
// order, and their error is the quantisation of the operands and the dropped
// low x low limb product: about one unit of 2^-61 of the largest sum a line
// could have, where a chain of FP64 operations rounds every partial sum to
// 2^-53.  (Those sums cancel: a smooth line's derivative is a hundredth of
// them, so the last bits count.)
//
//   values        |F| <= 2^59, pair sums |S| <= 2^60: hi 2^29 + lo,
//                 0 <= lo < 2^29
//   coefficients  c 2^60, |c| < 1: hi 2^29 + lo, -2^28 <= lo < 2^28; a row's
//                 magnitudes add up to less than 1 over the line's values
//                 (less than 1/2 over its pair sums)
//   accumulator   hh = sum Ch Xh, x = sum (Ch Xl + Cl Xh); result
//                 hh + (x >> 29) = sum C X / 2^58, at most 2^61, so that a
//                 node's three results add up in 64 bits.  |x| <= 2^60 + n 2^58
//                 for n <= 18 values, 2^59 + n 2^59 for n <= 10 pair sums.
//
// The same code compiles for the host, where tests check it.
#pragma once

#include <cstdint>

#include "sdg_df.cuh"

namespace sdg {

struct fixlimb {
  int32_t hi, lo;
};

constexpr int kFixLow = 29;  // bits of the low limb
constexpr int kFixMask = (1 << kFixLow) - 1;

SDG_HD fixlimb fix_split(int64_t x) {
  fixlimb r;
  r.hi = (int32_t)(x >> kFixLow);
  r.lo = (int32_t)((uint32_t)x & (uint32_t)kFixMask);
  return r;
}

// Limbs of a coefficient c 2^60 (|c| < 1): balanced low limb.
SDG_HD fixlimb fix_coef(int64_t c) {
  fixlimb r;
  r.hi = (int32_t)((c + (int64_t(1) << (kFixLow - 1))) >> kFixLow);
  r.lo = (int32_t)(c - ((int64_t)r.hi << kFixLow));
  return r;
}

// c 2^60 of a double |c| <= 1, truncated.
SDG_HD int64_t fix_unit(double c) {
  uint32_t hi, lo;
  d2words(c, hi, lo);
  const uint32_t e = (hi >> 20) & 0x7FFu;
  const uint64_t m = ((uint64_t)((hi & 0xFFFFFu) | 0x100000u) << 32 | lo) << 8;
  const int64_t r = e + 63 < 1023 || e > 1023 ? 0 : (int64_t)(m >> (1023 - e));
  return (int32_t)hi < 0 ? -r : r;
}

struct fixacc {
  int64_t hh, x;
};

// a b and a b + c as one 32 x 32 + 64 bit instruction: written out, since the
// compiler takes a limb it knows to be non-negative for an unsigned number and
// then forms a full 64-bit product (twice the instructions of a line).
SDG_HD int64_t fix_wide(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
  int64_t r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
#else
  return (int64_t)a * b;
#endif
}
SDG_HD int64_t fix_wide(int32_t a, int32_t b, int64_t c) {
#if defined(__CUDA_ARCH__)
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (int64_t)a * b + c;
#endif
}

SDG_HD void fix_mul(fixacc& a, fixlimb c, fixlimb v) {
  a.hh = fix_wide(c.hi, v.hi);
  a.x = fix_wide(c.lo, v.hi, fix_wide(c.hi, v.lo));
}
SDG_HD void fix_fma(fixacc& a, fixlimb c, fixlimb v) {
  a.hh = fix_wide(c.hi, v.hi, a.hh);
  a.x = fix_wide(c.lo, v.hi, fix_wide(c.hi, v.lo, a.x));
}
SDG_HD int64_t fix_sum(const fixacc& a) { return a.hh + (a.x >> kFixLow); }

// a b / 2^60 of two numbers below 2^60, two units off at most.
SDG_HD int64_t fix_times(int64_t a, int64_t b) {
  fixacc p;
  fix_mul(p, fix_split(a), fix_split(b));
  return fix_sum(p) >> (60 - 2 * kFixLow);
}

// a >> s, zero for s > 63 (the hardware shift clamps; C++ leaves it undefined).
SDG_HD uint64_t fix_shr(uint64_t a, uint32_t s) {
#if defined(__CUDA_ARCH__)
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(s));
  return r;
#else
  return s > 63 ? 0 : a >> s;
#endif
}

// x >> s for a non-negative s, the sign for s > 63 (as the hardware shifts).
SDG_HD int64_t fix_sar(int64_t x, int s) {
#if defined(__CUDA_ARCH__)
  int64_t r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
#else
  return x >> (s > 63 ? 63 : s);
#endif
}

// Exponent field of a double in place (bits 30..20 of the high word).
constexpr uint32_t kFixExp = 0x7FF00000u;

SDG_HD uint32_t fix_high(double x) {
  uint32_t hi, lo;
  d2words(x, hi, lo);
  return hi;
}

// A line's scale: E = the largest of its values' exponent fields and of its
// faces' less two (in place, at least zero).  With B = (E >> 20) - 1022 the
// line's values are F 2^(59 - B), |F| < 2^B, its faces a quarter of that.
SDG_HD int32_t fix_value_exp(double f) { return (int32_t)(fix_high(f) & kFixExp); }
SDG_HD int32_t fix_face_exp(double g) { return (int32_t)(fix_high(g) & kFixExp) - (2 << 20); }

// What the fixed-point path takes: B in [-700, 700).  Infinities and NaN lie
// above; a zero or subnormal value, whose significand is read as a normal
// one's, lies at least 300 bits below the line and aligns to zero.
SDG_HD bool fix_in_range(int32_t E) {
  return (uint32_t)E - (322u << 20) < (1400u << 20);
}
// A line's values within 2^6 of its largest are held exactly (59 bits of that for
// 53).  Where none but the largest lies within, a sum that does not see it (a zero
// on the diagonal) has fewer bits of the others than FP64.
constexpr int32_t kFixAlone = 6 << 20;
// The scale of a line that is to be formed in FP64: above the range.
constexpr int32_t kFixRefused = 2047 << 20;
// The scale of a line of zeros: the least of the range, marked in a bit that no
// other has, so that the line's exponent lies below all others and a node's sum
// is formed on the scale of its other lines.
constexpr int32_t kFixZeros = 322 << 20 | 1;
SDG_HD int fix_line_exp(int32_t E) { return (E >> 20) - 1022 - ((E & 1) << 11); }

// A value F 2^(59 - B), off by at most one unit (the magnitude truncated, a
// negative one then complemented, which is two instructions less than its
// negative: 2 % of a stage).  +0 gives zero, -0 minus one: products are formed by
// fix_product.  A face g / 4 2^(59 - B), its magnitude truncated: either zero gives
// zero.
SDG_HD double fix_product(double q, double u) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(q, u, 0.0);  // -0 + 0 = +0
#else
  return q * u + 0.0;
#endif
}
SDG_HD int64_t fix_align(double x, int32_t E) {
  uint32_t hi, lo;
  d2words(x, hi, lo);
  const uint32_t s = ((uint32_t)E - (hi & kFixExp)) >> 20;
  const uint64_t m = ((uint64_t)((hi & 0xFFFFFu) | 0x100000u) << 32 | lo) << 6;
  return (int64_t)fix_shr(m, s) ^ (int64_t)((int32_t)hi >> 31);
}
SDG_HD int64_t fix_align_signed(double x, int32_t E) {
  return fix_align(x, E) - ((int32_t)fix_high(x) >> 31);
}
SDG_HD int64_t fix_align_face(double g, int32_t E) {
  return fix_align_signed(g, E + (2 << 20));
}

// x 2^E, |x| < 2^63, to one unit of x and half an ulp of the result, for
// results in the normal range, and zero for zero; no FP64 operation and no
// conversion instruction, which run on the FP64 pipe, and no branch.  A negative
// x is complemented (a unit less).
SDG_HD double fix_to_double(int64_t x, int E) {
  const uint32_t xh = (uint32_t)(x >> 32), neg = (uint32_t)((int32_t)xh >> 31);
  uint32_t ah = xh ^ neg, al = (uint32_t)x ^ neg;
  // below 2^32: up by 31 bits
  const bool low = ah == 0u;
  ah = low ? al >> 1 : ah;
  al = low ? al << 31 : al;
  E = low ? E - 31 : E;
  // leading one to bit 62
#if defined(__CUDA_ARCH__)
  const int sh = __clz((int)ah) - 1;
  const uint32_t mh = __funnelshift_l(al, ah, sh);
#else
  const int sh = (ah ? __builtin_clz(ah) : 32) - 1;
  const uint32_t mh = (uint32_t)((((uint64_t)ah << 32 | al) << sh) >> 32);
#endif
  // rounded at bit 10; bit 52 of the rest (53 after a carry) adds one (two) to
  // the exponent field
  const uint64_t m = ((uint64_t)mh << 32 | (al << sh)) + 0x200u;
  const uint32_t hi = (uint32_t)(m >> 42) + ((uint32_t)(1023 + 61 + E - sh) << 20);
  return words2d(x == 0 ? 0u : hi | (xh & 0x80000000u), (uint32_t)(m >> 10));
}

}  // namespace sdg
