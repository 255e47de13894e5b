// cato_intdiv.cuh -- IEEE-754 binary64 division and square root, rounded to nearest even, on the
// integer pipe.
//
// GB300 runs FP64 arithmetic at 1/64 of the FP32 rate, and a division or square root costs
// several FP64 instructions there.  The integer and FP32 pipes have room to spare.  These
// routines get the exact IEEE result from integer arithmetic on the significands:
//   1. an FP32 seed y0 ~ 1 / b (division) or 1 / sqrt(a) (square root) of the operand's
//      significand truncated to 24 bits, from the hardware approximation (any seed within 2^-21
//      relative will do);
//   2. one Newton-Raphson step of third order in 64-bit fixed point, y1 = y0 (1 + e + e^2) for
//      1/b with e = 1 - b y0, and y1 = y0 (1 + e/2 + 3e^2/8) for 1/sqrt(a) with e = 1 - a y0^2
//      (J.-M. Muller et al., Handbook of Floating-Point Arithmetic, 2nd ed., 2018, sections 4.7
//      and 11.3: Newton-Raphson iterations for the reciprocal and the reciprocal square root);
//   3. the quotient a y1 (or the root a y1) from three 32 x 32-bit partial products of the
//      64 x 64-bit product, within 43 units of 2^-61 (29 units of 2^-60 for the root) of the exact
//      value, far inside the 128 units the next step allows, and its floor F as a significand;
//   4. the exact rounding decision: the sign of the integer remainder 2^k A - (2 F + 1) B
//      (division) or 2^k A - (2 F + 1)^2 (square root), computed modulo 2^64 because its
//      magnitude is below 2^63, decides between F and F + 1; neither has ties.
// Exact scalings by 2^-1, 2^-2, 2^-3 and 2 (scale_down, scale_up1) are exponent steps here.
// Operands that are zero, subnormal, infinite or NaN, negative square-root operands and quotients
// outside the normal range take the hardware instruction instead (the caller's fallback).
// The same source compiles for the host, with correctly rounded seeds that a test hook moves by a
// few ulps; a host test compares the routines bit for bit with the hardware division and square
// root.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define CATO_HD __host__ __device__ __forceinline__
#else
#define CATO_HD static inline
#endif

namespace cato {
namespace intdiv {

// The register pair itself, opaque to the compiler: from a plain bit cast it recognises the tests
// below (bits & 0x7fff... as |x|, (bits << 1) == 0 as x == 0) and turns them back into FP64-pipe
// instructions, which made 140 of the FP64 stage kernel's 340 per cell.
CATO_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
  uint64_t u;
  asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
  return u;
#else
  uint64_t u;
  memcpy(&u, &x, sizeof u);
  return u;
#endif
}
CATO_HD double double_of(uint64_t u) {
#ifdef __CUDA_ARCH__
  double x;
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(u));
  return x;
#else
  double x;
  memcpy(&x, &u, sizeof x);
  return x;
#endif
}
CATO_HD uint32_t fbits_of(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, sizeof u);
  return u;
#endif
}
CATO_HD float float_of(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, sizeof x);
  return x;
#endif
}
CATO_HD uint32_t umulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// floor(x y / 2^64) - d with 0 <= d < 3: the high half of a 64 x 64-bit product from three
// 32 x 32-bit products (the low x low product dropped, the cross products truncated)
CATO_HD uint64_t mulhi3(uint64_t x, uint64_t y) {
  const uint32_t xh = (uint32_t)(x >> 32), xl = (uint32_t)x, yh = (uint32_t)(y >> 32);
  const uint32_t yl = (uint32_t)y;
  return (uint64_t)xh * yh + (uint64_t)umulhi32(xh, yl) + (uint64_t)umulhi32(xl, yh);
}
// FP32 seeds y0 ~ 1/x and y0 ~ 1/sqrt(x) for x in [1, 4): on the device the single-instruction
// approximations (rcp.approx.ftz.f32, rsqrt.approx.ftz.f32).  The routines below are exact for
// any seed within 2^-21 relative of the true value (the error analysis keeps every fixed-point
// quantity inside 64 bits and the quotient within 4 units of its last bit); cato_gpu_check_divsqrt
// measures the hardware seeds' error over every input they get.  On the host the seeds are the
// correctly rounded values, moved by CATO_SEED_OFFSET units in the last place (a test hook that
// exercises seeds up to a few ulps off).
#if !defined(__CUDA_ARCH__) && defined(CATO_INTDIV_SEED_HOOK)
extern int seed_offset_ulps;
#define CATO_SEED_OFFSET seed_offset_ulps
#else
#define CATO_SEED_OFFSET 0
#endif
CATO_HD float recip_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return float_of(fbits_of(1.0f / x) + (uint32_t)CATO_SEED_OFFSET);
#endif
}
CATO_HD float rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return float_of(fbits_of((float)(1.0 / __builtin_sqrt((double)x))) + (uint32_t)CATO_SEED_OFFSET);
#endif
}

constexpr uint64_t kFrac = 0x000fffffffffffffULL;
constexpr uint64_t kHid = 0x0010000000000000ULL;

// y * 2^30 as an integer for an FP32 seed y in [0.5, 1]: its bits count units of 2^-24 from 0.5
// (a seed an ulp or two outside becomes another one as near)
CATO_HD uint32_t fixed30(float y) { return fbits_of(y) * 64u - 0x3e800000u * 64u; }

// y0 (1 + t) * 2^62 for y0 = Y0 / 2^30 and t = T / 2^80 (floor of the correction term)
CATO_HD uint64_t refine62(uint32_t Y0, int64_t T) {
  const int64_t Th = T >> 32;                 // floor(T / 2^32)
  const uint64_t Tl = (uint32_t)T;
  const int64_t yt32 = (int64_t)Y0 * Th + (int64_t)(((uint64_t)Y0 * Tl) >> 32);  // floor(Y0 T / 2^32)
  return ((uint64_t)Y0 << 32) + (uint64_t)(yt32 >> 16);
}

// RN(a / b) as bits for normal a, b; ok = false when an operand is not normal or the quotient
// is not normal (the bits are then meaningless).
//
// With A, B the 53-bit significands (a = A 2^(ea-1075), b = B 2^(eb-1075)):
//   y0 ~ 1 / fb, fb = b' = B / 2^52 truncated to 24 bits, |1 - fb y0| <= 2^-21, so that
//   e = 1 - b' y0 has |e| < 1.25 2^-21 (the bounds below hold up to |e| = 2^-19);
//   E = 2^80 e = -(B Y0 / 4) mod 2^64 (Y0 is a multiple of 4), |E| < 2^61;
//   T = E + Eh^2 / 2^16 (Eh = floor(E / 2^32)) = 2^80 (e + e^2) within 2^-66;
//   Y1 = 2^62 y0 (1 + T / 2^80): |Y1 - 2^62 / b'| < 2 (the omitted e^3 term: 2^-57 at most);
//   H ~ A 2^11 Y1 / 2^64 (mulhi3): |H - 2^61 A / B| < 43;
//   n = 1 when H < 2^61 (quotient below 1), and with the quotient's significand in [1, 2) as
//   Hn = 2^n H, An = 2^n A: Hn / 2^9 is within 0.17 of X = 2^52 An / B, so RN(X) is
//   F = floor(Hn / 2^9) or F + 1, decided by the sign of Z = 2^53 An - (2 F + 1) B (|Z| < 2^55,
//   and not 0: the odd 2 F + 1 >= 2^53 would divide A).  Where n is taken wrongly
//   (|H - 2^61| < 43), X lies within 0.17 of 2^52 or 2^53 and either choice rounds to the same
//   value.
// Y1 depends on b alone (recip62): quotients by the same divisor share it (quot_bits).
CATO_HD uint64_t recip62(uint64_t ub) {
  const uint64_t B = (ub & kFrac) | kHid;
  const float fb = float_of(0x3f800000u | (uint32_t)((ub & kFrac) >> 29));
  const uint32_t Y0 = fixed30(recip_seed(fb));
  const int64_t E = (int64_t)(0ULL - B * (uint64_t)(Y0 >> 2));
  const int32_t Eh = (int32_t)(E >> 32);
  const int64_t T = E + (((int64_t)Eh * Eh) >> 16);
  return refine62(Y0, T);
}
// quot_mag: |a / b|, for operands and a quotient known to be normal.
CATO_HD uint64_t quot_mag(uint64_t ua, uint64_t ub, uint64_t Y1) {
  const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
  const uint64_t A = (ua & kFrac) | kHid, B = (ub & kFrac) | kHid;
  const uint64_t H = mulhi3(A << 11, Y1);
  const uint32_t n = (uint32_t)(H >> 61) ^ 1u;
  const uint64_t F = H >> (9u - n);
  const int64_t Z = (int64_t)(((uint64_t)((uint32_t)A << (21u + n)) << 32) - (2 * F + 1) * B);
  // the exponents are subtracted in place; F in [2^52, 2^53): its leading bit and a carry go into
  // the exponent field
  const uint32_t Ef = (ha & 0x7ff00000u) - (hb & 0x7ff00000u) + ((1022u - n) << 20);
  return ((uint64_t)Ef << 32) + F + (Z > 0 ? 1u : 0u);
}
CATO_HD uint64_t quot_bits(uint64_t ua, uint64_t ub, uint64_t Y1, bool& ok) {
  const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
  const uint64_t q = quot_mag(ua, ub, Y1);
  const uint32_t ea = ha & 0x7ff00000u, eb = hb & 0x7ff00000u;
  // exponents 1..2046, and the quotient's from their difference, which cannot wrap
  const uint32_t d = ea - eb + (1022u << 20);
  ok = ea - 0x100000u < 2046u << 20 && eb - 0x100000u < 2046u << 20 && d - 0x100000u < 2044u << 20;
  return q ^ ((uint64_t)((ha ^ hb) & 0x80000000u) << 32);
}
CATO_HD uint64_t div_bits(uint64_t ua, uint64_t ub, bool& ok) {
  return quot_bits(ua, ub, recip62(ub), ok);
}

// RN(sqrt(a)) as bits for normal a > 0; ok = false otherwise.
//
// a = A2 2^(2m) with A2 = A or 2A in [2^52, 2^54), a'' = A2 / 2^52 in [1, 4):
//   y0 ~ 1 / sqrt(fa), fa = a'' truncated to 24 bits, |1 - fa y0^2| <= 2^-21, so that
//   e = 1 - a'' y0^2 has |e| < 1.5 2^-21 (the bounds below hold up to |e| = 2^-19);
//   E = 2^80 e = -floor(A2 Y0^2 / 2^32) mod 2^64 (within 2 units), |E| < 2^61;
//   T = E / 2 + 3 floor(Eh^2 / 2^19) = 2^80 (e/2 + 3e^2/8);  Y1 = 2^62 y0 (1 + T / 2^80), within
//   6 units (the omitted 5e^3/16 term: 2^-58.7 at most);
//   H ~ A2 2^10 Y1 / 2^64 (mulhi3): |H - 2^60 sqrt(a'')| < 29, inside the 128 the rounding
//   allows, so the root is F = floor(H / 2^8) or F + 1: the sign of
//   Z = 2^54 A2 - (2 F + 1)^2 (never 0), |Z| < 2^56.
CATO_HD uint64_t sqrt_bits(uint64_t ua, bool& ok) {
  const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu;
  const uint32_t odd = (ea & 1u) ^ 1u;  // the unbiased exponent ea - 1075 is odd
  const uint64_t A2 = ((ua & kFrac) | kHid) << odd;
  const float fa = float_of(((127u + odd) << 23) | (uint32_t)((ua & kFrac) >> 29));
  const uint32_t Y0 = fixed30(rsqrt_seed(fa));
  const uint64_t S = (uint64_t)Y0 * Y0;  // Y0^2 <= 2^60
  // floor(A2 S / 2^32) mod 2^64 from 32-bit halves (the carry out of the lowest product dropped)
  const uint32_t ah = (uint32_t)(A2 >> 32), al = (uint32_t)A2;
  const uint32_t sh = (uint32_t)(S >> 32), sl = (uint32_t)S;
  const uint64_t P = ((uint64_t)(ah * sh) << 32) + (uint64_t)ah * sl + (uint64_t)al * sh +
                     umulhi32(al, sl);
  const int64_t E = (int64_t)(0ULL - P);
  const int32_t Eh = (int32_t)(E >> 32);
  const int64_t T = (E >> 1) + 3 * (((int64_t)Eh * Eh) >> 19);
  const uint64_t Y1 = refine62(Y0, T);
  const uint64_t H = mulhi3(A2 << 10, Y1);
  const uint64_t F = H >> 8, N = 2 * F + 1;
  const int64_t Z = (int64_t)(((uint64_t)((uint32_t)A2 << 22) << 32) - N * N);
  ok = (ea - 1u < 2046u) && !(ua >> 63);
  const uint32_t Ef = 511u + ((ea - odd) >> 1);  // 1048 + (ea - 1075 - odd) / 2
  return (((uint64_t)Ef << 52) + F) + (Z > 0 ? 1u : 0u);  // F's leading bit adds one to Ef
}

// RN(a * b) as bits for normal a, b with a normal product; ok = false otherwise (zero, subnormal,
// infinite or NaN operands, products below the normal range or above the largest finite value;
// the bits are then meaningless).
//
// With A, B the 53-bit significands, the exact product P = A B (106 bits) is in [2^104, 2^106);
// t = 1 when P >= 2^105.  The rounded significand is M = floor(P / 2^(52+t)) plus one when the
// dropped bits exceed half a unit, or equal it with M odd (ties to even).  The dropped bits are
// left-aligned in a 64-bit word R, so that half a unit is 2^63.  M + 1 = 2^53 carries into the
// exponent field, and a carry out of the largest exponent gives the infinity that IEEE rounding
// to nearest gives.  Biased result exponent: ea + eb - 1023 + t.
CATO_HD uint64_t mul_bits(uint64_t ua, uint64_t ub, bool& ok) {
  const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu, eb = (uint32_t)(ub >> 52) & 0x7ffu;
  const uint64_t A = (ua & kFrac) | kHid, B = (ub & kFrac) | kHid;
#ifdef __CUDA_ARCH__
  const uint64_t hi = __umul64hi(A, B), lo = A * B;
#else
  const unsigned __int128 P = (unsigned __int128)A * B;
  const uint64_t hi = (uint64_t)(P >> 64), lo = (uint64_t)P;
#endif
  const uint32_t t = (uint32_t)(hi >> 41);  // P >= 2^105
  const uint64_t M = (hi << (12u - t)) | (lo >> (52u + t));
  const uint64_t R = lo << (12u - t);
  const uint64_t up = (R > 0x8000000000000000ULL || (R == 0x8000000000000000ULL && (M & 1u)))
                          ? 1u : 0u;
  const int32_t E = (int32_t)(ea + eb + t) - 1023;
  ok = (ea - 1u < 2046u) && (eb - 1u < 2046u) && (E >= 1) && (E <= 2046);
  const uint64_t sign = (ua ^ ub) & 0x8000000000000000ULL;
  return sign | ((((uint64_t)(uint32_t)(E - 1)) << 52) + M + up);
}

// x * 2^-K (K = 1, 2, 3) and x * 2, equal to the IEEE products: an exponent step when the
// result is normal; below the normal range the significand is shifted with round-to-nearest-even;
// 2x overflows to infinity; infinities and NaN pass through.
template <int K> CATO_HD double scale_down(double x) {
  const uint64_t u = bits_of(x), a = u & 0x7fffffffffffffffULL;
  const uint32_t e = (uint32_t)(a >> 52);
  if (e > (uint32_t)K) return e == 0x7ffu ? x : double_of(u - ((uint64_t)K << 52));
  const uint64_t n = e == 0u ? a : (((a & kFrac) | kHid) << (e - 1u));  // |x| = n 2^-1074
  const uint64_t q = n >> K, rem = n & ((1ULL << K) - 1ULL), h = 1ULL << (K - 1);
  const uint64_t r = q + ((rem > h || (rem == h && (q & 1ULL))) ? 1ULL : 0ULL);
  return double_of((u & 0x8000000000000000ULL) | r);
}
CATO_HD double scale_up1(double x) {
  const uint64_t u = bits_of(x), a = u & 0x7fffffffffffffffULL, s = u & 0x8000000000000000ULL;
  const uint32_t e = (uint32_t)(a >> 52);
  if (e == 0u) return double_of(s | (a << 1));  // zero or subnormal: exact
  if (e >= 0x7feu) return e == 0x7ffu ? x : double_of(s | 0x7ff0000000000000ULL);
  return double_of(u + (1ULL << 52));
}

// x + 1e-16, rounded to nearest even.  1e-16 = C 2^-106 with C = 0x1cd2b297d889bc; against an x of
// exponent field E >= 992 (2^-31) it is C 2^(969 - E) < 2^30 units of x's last place, never a tie
// (C's last set bit is its third).  Its rounded value is added to the bit pattern unless x is so
// near the ends of its binade that the sum could leave it.  ok = false: not computed here.
CATO_HD uint64_t add_1em16_bits(uint64_t x, bool& ok) {
  const uint32_t hi = (uint32_t)(x >> 32), s = (hi & 0x7fffffffu) - (992u << 20);
  ok = s < (1000u << 20) && ((hi + 1) & 0xfffffu) > 1u;
  const uint32_t sh = (s >> 20) + 1;
#ifdef __CUDA_ARCH__
  const uint32_t c = __funnelshift_rc(0xe69594beu, 0u, sh);
#else
  const uint32_t c = sh < 32 ? 0xe69594beu >> sh : 0u;
#endif
  const int32_t inc = (int32_t)((c + 1) >> 1), sg = (int32_t)hi >> 31;
  return x + (uint64_t)(int64_t)((inc ^ sg) - sg);
}

// 1 + x for x in [2^-32, 2), rounded to nearest even: the significand of x shifted to units of
// 2^-52 (from 1 up: its fraction, to units of 2^-51 above 2) by a multiplication, whose low word
// decides the rounding.  ok = false: not computed here (adding the 1 in place from 2 up takes more
// than it saves: 24.9 against 24.7 ms a step at 4096^2).
CATO_HD uint64_t one_plus_bits(uint64_t x, bool& ok) {
  const uint32_t hi = (uint32_t)(x >> 32), lo = (uint32_t)x, E = hi >> 20;
  ok = E - 991u <= 32u;
  const bool up = E == 1023u;
  const uint32_t p = 1u << (((up ? 1022u : E) - 991u) & 31u);
  const uint32_t mh = (hi & 0xfffffu) | (up ? 0u : 1u << 20);
  const uint64_t a = (uint64_t)lo * p, q = (uint64_t)mh * p + (a >> 32);
  const uint32_t odd = (uint32_t)q & 1u, round = (uint32_t)a > 0x80000000u - odd;
  return q + (((uint64_t)(up ? 0x40000000u : 0x3ff00000u) << 32) + round);
}

}  // namespace intdiv
}  // namespace cato
