// soft64.h -- correctly rounded FP64 division and square root on the integer
// pipe.
//
// GB300 takes one FP64 warp instruction every 64 cycles per SM sub-partition,
// and a division or square root is nine of them while the integer pipe idles.
// Both results are determined by exact integer arithmetic on the 53-bit
// significands, so they are formed there: a single-precision reciprocal
// (square root) estimate, one Newton step in fixed point, the quotient (root)
// in two digits of about 30 and 25 bits, each with its exact remainder modulo
// 2^64, and a last step that makes the result the floor of the true value.
// Neither a quotient nor a square root of 53-bit numbers lies midway between
// two doubles, so the bit below the last one decides the rounding.  (The
// digit-by-digit quotient with exact remainders is the schoolbook method;
// Newton's iteration for the reciprocal and the reciprocal square root, and
// the absence of midpoints, are textbook facts: Muller et al., Handbook of
// Floating-Point Arithmetic.)
//
// Cycles per warp and sub-partition, four warps each: division with two
// additions 682 -> 210, square root 557 -> 144.  One warp: 750 -> 550 and
// 626 -> 367.  FP64 SA, eight slices of 385x97: residual 1068 -> 767 us of an
// iteration, the iteration 2455 -> 2324 us.
//
// Operands outside the normal range, and results that could leave it, take
// the hardware operation, zeros excepted (a component of the velocity is 0
// over whole meshes).  Host code compiles the same functions, with an error
// of the estimates that a test can set.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define OT2D_HD __host__ __device__ __forceinline__
#else
#define OT2D_HD inline
#endif

namespace ot2d {
namespace soft64 {

#ifndef __CUDA_ARCH__
inline float& seed_error() { static float e = 0.f; return e; }   // relative, host tests only
#endif

OT2D_HD uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u; std::memcpy(&u, &x, 8); return u;
#endif
}
OT2D_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x; std::memcpy(&x, &u, 8); return x;
#endif
}
OT2D_HD uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u; std::memcpy(&u, &x, 4); return u;
#endif
}
OT2D_HD float from_fbits(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x; std::memcpy(&x, &u, 4); return x;
#endif
}
OT2D_HD float rcp_est(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return (1.0f / x) * (1.0f + seed_error());
#endif
}
OT2D_HD float rsqrt_est(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return (float)(1.0 / std::sqrt((double)x)) * (1.0f + seed_error());
#endif
}
OT2D_HD uint64_t mulw(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
OT2D_HD int64_t mulws(int32_t a, int32_t b) { return (int64_t)a * b; }

// An estimate r in [0.5, 1] as an integer multiple of 2^-23 below 2^23: r is
// moved down by 2^-21 (so it stays below 1) and added to 1, which leaves it
// in the low bits of the sum.  At most 1.5 * 2^-21 from r.
OT2D_HD uint32_t fixed23(float r) { return fbits((r - 4.76837158e-07f) + 1.0f) & 0x7fffffu; }

// a / b, rounded to nearest even
OT2D_HD double div(double a, double b) {
  const uint64_t ua = bits(a), ub = bits(b);
  const int ea = (int)((uint32_t)(ua >> 52) & 0x7ff), eb = (int)((uint32_t)(ub >> 52) & 0x7ff);
  // both normal, and the result (exponent ea - eb + 1023, or one less) too
  if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u || (unsigned)(ea - eb + 1021) >= 2043u)
    return ((ua << 1) == 0 && (unsigned)(eb - 1) < 2046u) ? from_bits((ua ^ ub) & 0x8000000000000000ull) : a / b;
  const uint64_t ma = (ua & 0xfffffffffffffull) | 0x10000000000000ull, mb = (ub & 0xfffffffffffffull) | 0x10000000000000ull;
  // r = 1 / b with b in [1, 2): 23 bits, within 2^-20 of it
  const uint32_t r0 = fixed23(rcp_est(from_fbits(0x3f800000u | ((uint32_t)(ub >> 29) & 0x7fffffu))));
  // Newton: b r0 in units of 2^-54, its distance from 1 in units of 2^-50,
  // then r in units of 2^-32, within 2^-30
  const uint32_t bh = (uint32_t)(mb >> 21), bl = (uint32_t)(mb << 11);
  const uint64_t t = mulw(bh, r0) + (mulw(bl, r0) >> 32);
  const int32_t e = (int32_t)((int64_t)((1ull << 54) - t) >> 4);
  const uint32_t r = (r0 << 9) + (uint32_t)(int32_t)(mulws((int32_t)r0, e) >> 41);
  // first digit: q1 about ma 2^30 / mb, and its remainder (a few mb)
  const uint32_t q1 = (uint32_t)(mulw((uint32_t)(ma >> 21), r) >> 33);
  const uint64_t q1mb = mulw(q1, (uint32_t)mb) + ((uint64_t)(q1 * (uint32_t)(mb >> 32)) << 32);
  const int64_t rem1 = (int64_t)((ma << 30) - q1mb);
  // second digit: q2 about rem1 2^25 / mb
  const int32_t q2 = (int32_t)(((rem1 >> 27) * (int64_t)r) >> 32);
  int64_t rem = (int64_t)(((uint64_t)rem1 << 25) - (uint64_t)(int64_t)q2 * mb);
  uint64_t q = ((uint64_t)q1 << 25) + (uint64_t)(int64_t)q2;
  // make q the floor of ma 2^55 / mb: the digits leave it within a few units
  if (rem < 0) { rem += (int64_t)mb; --q; }
  if (rem < 0) { rem += (int64_t)mb; --q; }
  if (rem >= (int64_t)mb) { rem -= (int64_t)mb; ++q; }
  if (rem >= (int64_t)mb) { rem -= (int64_t)mb; ++q; }
  // 2^54 <= q < 2^56: 53 bits and the deciding one
  const int big = (int)(q >> 55);
  q >>= 1 + big;
  const uint64_t m = (q >> 1) + (q & 1);
  const uint64_t ex = (uint64_t)(uint32_t)(ea - eb + 1021 + big) << 52;
  return from_bits(((ua ^ ub) & 0x8000000000000000ull) | (ex + m));
}

// sqrt(x), rounded to nearest even
OT2D_HD double sqrt_rn(double x) {
  const uint64_t ux = bits(x);
  const uint32_t ex = (uint32_t)(ux >> 52);                    // sign and exponent
  if (ex - 1u >= 2046u) return ux == 0 ? x : ::sqrt(x);        // zero, subnormal, infinite, NaN or negative
  // x = m 2^-52 4^h, m in [2^52, 2^54)
  const uint32_t odd = (ex & 1) ^ 1;                           // 1023 + odd exponent
  const uint64_t m = ((ux & 0xfffffffffffffull) | 0x10000000000000ull) << odd;
  // y = 1 / sqrt(m 2^-52) in (0.5, 1]: 23 bits, then Newton
  const float f = from_fbits((0x3f800000u + (odd << 23)) | ((uint32_t)(ux >> 29) & 0x7fffffu));
  const uint32_t y0 = fixed23(rsqrt_est(f));
  // x y0^2 in units of 2^-54 (y0^2 in units of 2^-46), its distance from 1 in
  // units of 2^-48, then y in units of 2^-32
  const uint64_t yy = mulw(y0, y0);                            // below 2^46
  const uint64_t mh = m >> 22;                                 // units of 2^-30, below 2^32
  const uint32_t yh = (uint32_t)(yy >> 14);                    // units of 2^-32
  const uint64_t t = mulw((uint32_t)mh, yh);                   // units of 2^-62
  const int32_t e = (int32_t)((int64_t)((1ull << 62) - t) >> 14);
  const uint32_t y = (y0 << 9) + (uint32_t)(int32_t)(mulws((int32_t)y0, e) >> 40);
  // first digit: s1 about sqrt(x) 2^30, remainder in units of 2^-60
  const uint32_t s1 = (uint32_t)(mulw((uint32_t)mh, y) >> 32);
  const int64_t rem1 = (int64_t)((m << 8) - mulw(s1, s1));
  // second digit: the root in units of 2^-53
  const int32_t s2 = (int32_t)(((rem1 >> 4) * (int64_t)y) >> 36);
  uint64_t s = ((uint64_t)s1 << 23) + (uint64_t)(int64_t)s2;
  // make s the floor: 0 <= m 2^54 - s^2 <= 2 s
  int64_t rem = (int64_t)((m << 54) - s * s);
  if (rem < 0) { --s; rem += (int64_t)(2 * s + 1); }
  if (rem < 0) { --s; rem += (int64_t)(2 * s + 1); }
  if (rem > (int64_t)(2 * s)) { rem -= (int64_t)(2 * s + 1); ++s; }
  if (rem > (int64_t)(2 * s)) { rem -= (int64_t)(2 * s + 1); ++s; }
  const uint64_t r = (s >> 1) + (s & 1);
  // biased exponent of the result less one: the significand's leading bit adds it
  return from_bits(((uint64_t)(((ex + 1023u - odd) >> 1) - 1) << 52) + r);
}

}  // namespace soft64
}  // namespace ot2d
