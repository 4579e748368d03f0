// IEEE double products and quotients, rounded to nearest even, computed on the
// integer pipe from the operands' bits.
//
// GB300 issues one FP64 instruction per SM and 16 clocks (2 lanes per clock);
// in those clocks its four schedulers can issue 64 other instructions. In
// place of the 7 or more FP64 instructions of an IEEE division (114 clocks of
// the SM measured per warp instruction) the quotient below takes about 66 issue
// slots, and in place of the 3 of a division by a row constant with its
// reciprocal (48 clocks) about 40. So in kernels bound by the FP64 unit the
// quotients go to the integer pipe and the additions stay on the FP64 unit.
//
// Every function takes magnitudes (bit patterns without the sign) of normal
// numbers and returns the magnitude of a result that must be normal too:
// callers test the operands' exponents (in_window) and leave everything else
// to the FP64 unit. Plain C++, so that the same text runs on the host.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define SIG_FN __host__ __device__ __forceinline__
#else
#define SIG_FN static inline
#endif

namespace sw2g {

constexpr uint64_t SIG_ONE = 1ULL << 52;
constexpr uint32_t SIG_EXP = 0x7ff00000u;
constexpr uint32_t SIG_BIAS = 1023u << 20;

// |x| in [2^-127, 2^129), x given by its upper word: operands for which the
// chains of the kernels have normal intermediate results.
SIG_FN bool in_window(uint32_t hi) { return ((hi + 0x08000000u) & 0x70000000u) == 0x40000000u; }

SIG_FN uint64_t sig_of(uint64_t a) { return (a & (SIG_ONE - 1)) | SIG_ONE; }
SIG_FN uint32_t sig_exp(uint64_t a) { return (uint32_t)(a >> 32) & SIG_EXP; }
// m in [2^52, 2^53] with the exponent field `e20` (in place, bits 20..30) of a
// leading one at bit 52; m = 2^53 carries into the exponent.
SIG_FN uint64_t sig_pack(uint64_t m, uint32_t e20) { return m + ((uint64_t)(e20 - (1u << 20)) << 32); }

// Upper 64 bits of a 64 x 64 bit product by four 32 x 32 -> 64 multiply-adds;
// mid: the upper half of the lower 64 bits, low: the rest.
SIG_FN uint64_t sig_mulhi(uint64_t a, uint64_t b, uint32_t* mid, uint32_t* low) {
  const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
  const uint64_t p = (uint64_t)a0 * b0;
  const uint64_t m1 = (uint64_t)a0 * b1 + (p >> 32);
  const uint64_t m2 = (uint64_t)a1 * b0 + (uint32_t)m1;
  *mid = (uint32_t)m2;
  *low = (uint32_t)p;
  return (uint64_t)a1 * b1 + (m1 >> 32) + (m2 >> 32);
}

// |a * b| * 2^k, k20 = k << 20. The 106-bit product is taken to t = P >> 51 in
// [2^53, 2^55): one or two bits below the result's last place.
SIG_FN uint64_t sig_mul(uint64_t a, uint64_t b, uint32_t k20 = 0) {
  uint32_t mid, low;
  const uint64_t t = sig_mulhi(sig_of(a) << 11, sig_of(b) << 2, &mid, &low);
  const uint32_t sh = 1u + ((uint32_t)(t >> 32) >> 22);
  uint64_t m = (t + sh) >> sh;
  if ((mid | low) == 0 && ((uint32_t)t & (2 * sh - 1)) == sh) m &= ~1ULL;  // a tie goes to even
  return sig_pack(m, sig_exp(a) + sig_exp(b) + k20 - SIG_BIAS + ((sh - 1) << 20));
}

// |(a * b) * c|, rounded after each product, where sig_mul3_far does not say
// that a, b (a zero too) or a product is not a normal number, or the result not in
// 2^-921 .. 2^121. For c in 2^-902 .. 2^102 and |a * c| at most 2^101: with c's
// range, a result in that window leaves no room for an a * b outside the normal
// range, and with |a * c|'s none for a b below it. ha, hb, hc: upper words.
SIG_FN bool sig_mul3_far(uint32_t ha, uint32_t hb, uint32_t hc) {
  const uint32_t ea = ha >> 20, e = ea + (hb >> 20) + (hc >> 20);
  return ea - 1 >= 2046u || e - 2148u >= 1042u;
}
SIG_FN uint64_t sig_mul3(uint64_t a, uint64_t b, uint64_t c) { return sig_mul(sig_mul(a, b), c); }

// The last step of a quotient N / mb in [1, 2) (mb: 53 bits): t = floor(N/mb *
// 2^53) or, where `unsure`, possibly one less than it; the quotient of two
// doubles is never a tie, so t's last bit (the half) decides the rounding, and
// only an even t can be wrong by it. The remainder has at most 54 bits, so
// its low 64 bits give its sign.
SIG_FN uint64_t sig_round_quotient(uint64_t t, bool unsure, uint64_t N, uint64_t mb) {
  if (unsure) {
    if ((int64_t)((N << 53) - (t + 1) * mb) >= 0) t += 1;
  }
  return (t + 1) >> 1;
}

// floor(2^127 / (b's significand at bit 63)), at most 2^64 - 1: the
// reciprocal of a divisor known in advance (host side).
static inline uint64_t sig_recip(uint64_t b) {
  const unsigned __int128 y = ((unsigned __int128)1 << 127) / (sig_of(b) << 11);
  return (y >> 64) ? ~0ULL : (uint64_t)y;
}

// |a / b| with y = sig_recip(b). The estimate 2N*y/2^64 is at most 2^-9 below
// N/mb*2^53 (y is at most one unit short, 2N < 2^55).
SIG_FN uint64_t sig_div_known(uint64_t a, uint64_t b, uint64_t y) {
  const uint64_t ma = sig_of(a), mb = sig_of(b);
  const bool ge = ma >= mb;
  const uint64_t N = ge ? ma : ma + ma;
  uint32_t mid, low;
  const uint64_t t = sig_mulhi(N + N, y, &mid, &low);
  const uint64_t m = sig_round_quotient(t, mid >= 0xff800000u, N, mb);
  return sig_pack(m, sig_exp(a) - sig_exp(b) + SIG_BIAS - (ge ? 0u : 1u << 20));
}

// 1/f of a float in (1, 2], within one ulp (2^-24).
SIG_FN float sig_rcp(float f) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return r;
#else
  return 1.0f / f;
#endif
}
union SigFloat {
  float f;
  uint32_t u;
};
SIG_FN uint32_t sig_mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// |a / b|, by long division in three digits of about 20 bits. y is the
// reciprocal of b's leading 24 bits rounded up (at most 2^-23 above b in
// [1, 2)), less three ulps of 2^-24. With the approximation within one ulp it
// is below 1/b, by a factor of at most 1 - 9*2^-24, or, where it falls below 1/2 (f =
// 2), whose ulps count double here, 1 - 11*2^-24. So every digit comes out low and
// every remainder is positive: below 1410, 971 and 670 units of the digit's place
// (e -> e*2^20*11*2^-24 + 2, from 2*2^30*11*2^-24 + 2), the first below 2^64. The
// sum of the digits is at most 670 units of 2^-70 below the quotient; the rounding
// test allows 700.
SIG_FN uint64_t sig_div(uint64_t a, uint64_t b) {
  const uint64_t ma = sig_of(a), mb = sig_of(b);
  SigFloat f;
  f.u = (0x3f800000u | ((uint32_t)(mb >> 29) & 0x7fffffu)) + 1u;
  f.f = sig_rcp(f.f);
  const uint32_t y = (f.u << 8) + (0x80000000u - 0x300u);  // units of 2^-32; a sum: it carries on below 1/2
  const bool ge = ma >= mb;
  const uint64_t N = ge ? ma : ma + ma;
  const uint32_t q1 = sig_mulhi32((uint32_t)(N >> 22), y);  // units of 2^-30
  const uint64_t r1 = (N << 30) - (uint64_t)q1 * mb;
  const uint32_t q2 = sig_mulhi32((uint32_t)(r1 >> 32), y);  // units of 2^-50
  const uint64_t r2 = (r1 << 20) - (uint64_t)q2 * mb;
  const uint32_t q3 = sig_mulhi32((uint32_t)(r2 >> 32), y);  // units of 2^-70
  const uint64_t t = ((uint64_t)q1 << 23) + ((uint64_t)q2 << 3) + (q3 >> 17);
  const uint64_t m = sig_round_quotient(t, (q3 & 0x1ffffu) >= 0x20000u - 700u, N, mb);
  return sig_pack(m, sig_exp(a) - sig_exp(b) + SIG_BIAS - (ge ? 0u : 1u << 20));
}

// How many of the operations above give another result than the product and
// the quotient of a and b, with y = sig_recip of b's bits (none where an operand
// or result is not a normal number).
union SigDouble {
  double d;
  uint64_t u;
};
SIG_FN uint64_t sig_mag(double x) {
  SigDouble v;
  v.d = x;
  return v.u & 0x7fffffffffffffffULL;
}
SIG_FN bool sig_normal(uint64_t a) { return (a >> 52) - 1 < 2046; }
SIG_FN int sig_mismatches(double a, double b, uint64_t y) {
  const uint64_t A = sig_mag(a), B = sig_mag(b), q = sig_mag(a / b), p = sig_mag(a * b);
  int n = 0;
  if (!sig_normal(A) || !sig_normal(B)) return 0;
  if (sig_normal(q)) n += (sig_div(A, B) != q) + (sig_div_known(A, B, y) != q);
  if (sig_normal(p)) {
    n += sig_mul(A, B) != p;
    if (sig_normal(p - SIG_ONE)) n += sig_mul(A, B, 0xfff00000u) != p - SIG_ONE;
  }
  return n;
}
// Whether sig_rcp(f), 1 < f <= 2, is within 2^-24 of 1/f (the product has 48 bits, the difference fewer).
SIG_FN bool sig_rcp_close(float f) {
  const double e = (double)sig_rcp(f) * (double)f - 1.0;
  return (e < 0 ? -e : e) <= 0x1p-24 * (double)f;
}

}  // namespace sw2g
