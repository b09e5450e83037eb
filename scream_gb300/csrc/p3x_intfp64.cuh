/*
 * FP64 operations on the integer pipes.
 *
 * The FP64 pipe of sm_103a takes a warp instruction every 16 SM cycles, so
 * one FP64 instruction costs as much pipe time as 64 issue slots of the SM's
 * four schedulers, while the integer and FP32 pipes of the FP64 kernels are
 * nearly idle.  A composite FP64 operation is therefore cheaper as integer
 * arithmetic on the significands.  Measured on one GB300 (SM cycles per warp
 * instruction with the SM full of warps; latency of a lone warp in cycles):
 *   FP64 add, multiply, FMA, conversion   15.5-18    ~100
 *   FP64 division                         131        564
 *   ddiv_int inlined / called             22 / 28    192 / 287
 */
#pragma once

#include <cstdint>
#include <cstring>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

namespace p3x {
namespace dev {

#ifdef __CUDACC__
#define P3X_HD __host__ __device__ __forceinline__
#define P3X_HD_NOINLINE static __host__ __device__ __noinline__
#else
#define P3X_HD inline
#define P3X_HD_NOINLINE static
#endif

P3X_HD uint64_t d_bits(double x) {
#ifdef __CUDA_ARCH__
  return uint64_t(__double_as_longlong(x));
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
P3X_HD double d_from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(u));
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
P3X_HD uint32_t mulhi_u32(uint32_t a, uint32_t b) { return uint32_t((uint64_t(a) * b) >> 32); }

/* 2^24 / f for a float f in [1, 2] given by its bits, as an integer in
 * [2^23 - 3, 2^24 - 1]: the FP32 reciprocal's significand less 2 units, so
 * that it never exceeds 2^24 / b for a b that rounds to f (the approximate
 * reciprocal is within one unit in the last place of 1/f, and the rounding of
 * b moves 1/b by at most one unit).  It falls short of 2^24 / b by at most 4
 * units near b = 1 and 3.3 near b = 2: a relative error below 2^-21.2. */
P3X_HD uint32_t rcp_seed(uint32_t fbits) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
  return __float_as_uint(r) - 0x3e800002u;
#else
  float f, r;
  std::memcpy(&f, &fbits, 4);
  r = 1.0f / f;
  uint32_t u;
  std::memcpy(&u, &r, 4);
  return u - 0x3e800002u;
#endif
}

/* a / b, rounded to nearest as IEEE division: the operands that the integer
 * sequence does not take (subnormals, infinities, NaN, b = 0, a quotient near
 * or outside the normal range, and the one in about a thousand whose last
 * bits leave the rounding open). */
P3X_HD_NOINLINE double ddiv_general(double a, double b) { return a / b; }

/* a / b on the integer pipes, the same double as the FP64 division.
 *
 * The 53-bit significands A and B give Q = A / B in (1/2, 2) by long division
 * in three digits from one FP32 reciprocal seed R <= 2^24 / (B / 2^52): each
 * digit is the high word of (leading remainder bits) x R, never above the
 * true one, and its exact remainder feeds the next.
 *   q1 ~ Q 2^30,              rem1 = A 2^30 - q1 B        in [0, 2^63)
 *   q2 ~ (rem1 / B) 2^19,     rem2 = rem1 2^19 - q2 B     in [0, 2^61)
 *   q3 ~ (rem2 / B) 2^19
 * S = q1 2^33 + q2 2^14 + (q3 >> 5) is then Q 2^63 less under 2 units (the
 * cube of the seed's error, 2^-63.6, and the truncations), and a quotient of
 * doubles is never half way between two doubles, so the nearest double follows
 * from S except where its bits below the last place are the ones just under
 * one half: one quotient in 1024, which takes the FP64 division. */
P3X_HD double ddiv_int(double a, double b) {
  const uint64_t ua = d_bits(a), ub = d_bits(b);
  const uint32_t ah = uint32_t(ua >> 32), al = uint32_t(ua), bh = uint32_t(ub >> 32), bl = uint32_t(ub);
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  const uint32_t mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t A = (uint64_t(mah) << 32) | al, B = (uint64_t(mbh) << 32) | bl;
  /* B / 2^52 rounded to the nearest float */
  const uint32_t R7 = rcp_seed((uint32_t((ub << 12) >> 40) + 0x7f000001u) >> 1) << 7;
  const uint32_t q1 = mulhi_u32(uint32_t(A >> 21), R7);
  const uint64_t rem1 = (A << 30) - B * q1;
  const uint32_t q2 = mulhi_u32(uint32_t(rem1 >> 32), R7);
  const uint64_t rem2 = (rem1 << 19) - B * q2;
  const uint32_t q3 = mulhi_u32(uint32_t(rem2 >> 32), R7);
  uint64_t S = (uint64_t(q1) << 33) + (uint64_t(q2) << 14) + (q3 >> 5);
  const uint32_t low = uint32_t(S >> 63) ^ 1u; /* 1: Q < 1 */
  S <<= low;
  const uint32_t er = ea - eb + 1022u - low; /* the result's exponent field less one */
  const uint32_t round = (uint32_t(S) >> 10) & 1u;
  const uint64_t r = (uint64_t(er) << 52) + (S >> 11) + round;
  const double res = d_from_bits(r ^ (uint64_t(sign) << 32));
  const bool open = (uint32_t(S) & 0x7feu) == 0x3feu;
  if (ea - 1u < 2046u && eb - 1u < 2046u && er - 1u < 2043u && !open) return res;
  if ((ua << 1) == 0 && eb - 1u < 2046u) return d_from_bits(uint64_t(sign) << 32); /* 0 / b */
  return ddiv_general(a, b);
}

}  // namespace dev
}  // namespace p3x
