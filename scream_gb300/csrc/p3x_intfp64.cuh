/*
 * FP64 operations on the integer pipes.
 *
 * The FP64 pipe of sm_103a takes a warp instruction every 16 SM cycles, so
 * one FP64 instruction costs as much pipe time as 64 issue slots of the SM's
 * four schedulers, while the integer and FP32 pipes of the FP64 kernels are
 * nearly idle.  A composite FP64 operation is therefore cheaper as integer
 * arithmetic on the significands.  Measured on one GB300 (SM cycles per warp
 * instruction with the SM full of warps; latency of a lone warp in cycles):
 *   FP64 add, multiply, FMA, conversion      15.5-18    ~100
 *   FP64 division                            131        564
 *   ddiv_int inlined / called                22 / 28    192 / 287
 *   raw_quotient (not rounded)               16
 *   64-bit high product, exact / mulhi_add   8.9 / 5.8  29
 *   log10 / log2 in Q57                      553 / 35
 *   cbrt / cbrt_int                          227 / 73
 *   pow / pow_int                            1499 / 76
 *   ice-table position / one column of it and its double (14 FP64 operations)
 *                                            17 / 42 (224)
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
/* IEEE comparisons of any double x with a constant c > 0 on the integer pipes:
 * the bit patterns as unsigned numbers are 0 to kInf for +0 to +infinity, 2^63
 * to 2^63 + kInf for -0 to -infinity, and the NaNs of either sign lie behind
 * those, so each test is one or two ranges (false for a NaN). */
constexpr uint64_t kInfPattern = 0x7ff0000000000000ull, kSignPattern = 0x8000000000000000ull;
P3X_HD bool ieee_gt(double x, double c) { return d_bits(x) - d_bits(c) - 1 < kInfPattern - d_bits(c); }
P3X_HD bool ieee_ge(double x, double c) { return d_bits(x) - d_bits(c) <= kInfPattern - d_bits(c); }
P3X_HD bool ieee_lt(double x, double c) {
  return d_bits(x) < d_bits(c) || d_bits(x) - kSignPattern <= kInfPattern;
}
/* x < 0 */
P3X_HD bool ieee_neg(double x) { return d_bits(x) - kSignPattern - 1 < kInfPattern; }

P3X_HD int64_t mulhi_s64(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return int64_t((__int128(a) * b) >> 64);
#endif
}
P3X_HD uint64_t mulhi_u64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return uint64_t((static_cast<unsigned __int128>(a) * b) >> 64);
#endif
}
P3X_HD int32_t mulhi_s32(int32_t a, int32_t b) { return int32_t((int64_t(a) * b) >> 32); }
/* acc + (a b >> 64), good to 4 units: the product of the low words is left
 * out, and the cross products lose the low word's last bit, which makes that
 * word a positive signed one.  Five instructions of the multiplier pipe, where
 * the exact high product takes a dozen, half of them on the adder pipe.  For
 * products with bits to spare below the last one that counts. */
P3X_HD int64_t mulhi_add(int64_t acc, int64_t a, int64_t b) {
  const int32_t ah = int32_t(a >> 32), bh = int32_t(b >> 32);
  const int32_t al = int32_t(uint32_t(a) >> 1), bl = int32_t(uint32_t(b) >> 1);
#ifdef __CUDA_ARCH__
  int32_t x;
  asm("mul.hi.s32 %0, %1, %2;" : "=r"(x) : "r"(ah), "r"(bl));
  asm("mad.hi.s32 %0, %1, %2, %3;" : "=r"(x) : "r"(bh), "r"(al), "r"(x));
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(acc) : "r"(ah), "r"(bh), "l"(acc));
  asm("mad.wide.s32 %0, %1, 2, %2;" : "=l"(acc) : "r"(x), "l"(acc));
  return acc;
#else
  return acc + int64_t(ah) * bh + 2 * int64_t(mulhi_s32(ah, bl) + mulhi_s32(bh, al));
#endif
}
P3X_HD int clz_u64(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __clzll(static_cast<long long>(x));
#else
  return x ? __builtin_clzll(x) : 64;
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

/* The quotient A / B of two 53-bit significands (bit 52 set), in units of
 * 2^-63, less under 2 units: S in [2^62, 2^64).
 *
 * Long division in three digits from one FP32 reciprocal seed R <= 2^24 /
 * (B / 2^52): each digit is the high word of (leading remainder bits) x R,
 * never above the true one, and its exact remainder feeds the next.
 *   q1 ~ Q 2^30,              rem1 = A 2^30 - q1 B        in [0, 2^63)
 *   q2 ~ (rem1 / B) 2^19,     rem2 = rem1 2^19 - q2 B     in [0, 2^61)
 *   q3 ~ (rem2 / B) 2^19
 * S = q1 2^33 + q2 2^14 + (q3 >> 5): the cube of the seed's error, 2^-63.6, and
 * the truncations stay below 2 units. */
P3X_HD uint64_t sig_quotient(uint64_t A, uint64_t B) {
  /* B / 2^52 rounded to the nearest float */
  const uint32_t R7 = rcp_seed((uint32_t((B << 12) >> 40) + 0x7f000001u) >> 1) << 7;
  const uint32_t q1 = mulhi_u32(uint32_t(A >> 21), R7);
  const uint64_t rem1 = (A << 30) - B * q1;
  const uint32_t q2 = mulhi_u32(uint32_t(rem1 >> 32), R7);
  const uint64_t rem2 = (rem1 << 19) - B * q2;
  const uint32_t q3 = mulhi_u32(uint32_t(rem2 >> 32), R7);
  return (uint64_t(q1) << 33) + (uint64_t(q2) << 14) + (q3 >> 5);
}

/* a / b on the integer pipes, the same double as the FP64 division.  A
 * quotient of doubles is never half way between two doubles, so the nearest
 * double follows from sig_quotient except where its bits below the last place
 * are the ones just under one half: one quotient in 1024, which takes the FP64
 * division. */
P3X_HD double ddiv_int(double a, double b) {
  const uint64_t ua = d_bits(a), ub = d_bits(b);
  const uint32_t ah = uint32_t(ua >> 32), bh = uint32_t(ub >> 32);
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  uint64_t S = sig_quotient((uint64_t((ah & 0xfffffu) | 0x100000u) << 32) | uint32_t(ua),
                            (uint64_t((bh & 0xfffffu) | 0x100000u) << 32) | uint32_t(ub));
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

/* ------------------------------------------------------------------ */
/* logarithm, exponential, powers in 64-bit fixed point                */
/* ------------------------------------------------------------------ */
/* Fixed-point values are written Qn: an integer in units of 2^-n. */

/* Tables of the functions below, 128 intervals each: r is 2^32 / c for the
 * interval's midpoint c, rounded, and nlog2 = -log2(r / 2^32) in Q62; exp2
 * holds 2^((j + 1/2) / 128) in Q62.  They are static data of the module (3 KB
 * per translation unit), so no launch depends on a context or an upload. */
struct alignas(16) Log2Entry {
  uint32_t r, pad;
  int64_t nlog2;
};
struct FixTables {
  Log2Entry log2[128];
  int64_t exp2[128];
};
#ifdef __CUDACC__
static __device__ const FixTables kFixTables =
#include "p3x_fixtables.inc"
    ;
#else
static const FixTables kFixTables =
#include "p3x_fixtables.inc"
    ;
#endif

/* log2 of M63 / 2^63 for a significand with bit 63 set, in Q62.  With r ~ 1 / c
 * the table leaves z = r M63 / 2^63 - 1, |z| < 2^-8, exact to 2^-63, and
 * ln(1 + z) = z - z^2 (1/2 - z (1/3 - z (1/4 - z (1/5 - z / 6)))) is cut off
 * below 2^-58; the inner terms need 32 bits only.  Error below 2^-57. */
P3X_HD int64_t log2_sig(uint64_t M63, const FixTables* t) {
  const Log2Entry* en = &t->log2[uint32_t(M63 >> 56) & 127u];
#ifdef __CUDA_ARCH__
  const uint4 ev = __ldg(reinterpret_cast<const uint4*>(en));
  const uint32_t r = ev.x;
  const int64_t nl = int64_t((uint64_t(ev.w) << 32) | ev.z);
#else
  const uint32_t r = en->r;
  const int64_t nl = en->nlog2;
#endif
  const uint64_t P = (M63 >> 32) * r + ((uint64_t(uint32_t(M63)) * r) >> 32);
  const int64_t z = int64_t(P - (1ull << 63)); /* Q63 */
  const int64_t z8 = z << 8;                    /* Q71 */
  const int32_t zs = int32_t(z >> 24);          /* Q39 */
  constexpr int32_t k6 = int32_t((1ll << 31) / 6), k5 = int32_t((1ll << 31) / 5), k4 = 1 << 29;
  constexpr int64_t k3 = (1ll << 62) / 3, k2 = 1ll << 61, kLog2e = 6653256548922161245ll; /* log2(e) Q62 */
  const int32_t t4 = k5 - (mulhi_s32(zs, k6) >> 7);
  const int32_t t3 = k4 - (mulhi_s32(zs, t4) >> 7);
  const int64_t t2 = k3 - ((int64_t(zs) * t3) >> 8);
  const int64_t t1 = k2 - (mulhi_add(0, z8, t2) >> 7);
  const int64_t u = mulhi_add(0, z8, t1);      /* z t1, Q69 */
  const int64_t v = mulhi_add(0, z8, u << 3);  /* z^2 t1, Q79 */
  const int64_t ln = z8 - (v >> 8);            /* Q71 */
  return nl + (mulhi_add(0, ln, kLog2e) >> 7);
}

/* 2^F for F in [0, 1) given in Q64: the significand in Q62, error below
 * 2^-60.  2^(1/256 + j/128) from the table times e^g, |g| < 2^-8.5, with
 * e^g - 1 = g + g^2 (1/2 + g (1/6 + g (1/24 + g (1/120 + g / 720)))). */
P3X_HD int64_t exp2_sig(uint64_t F, const FixTables* t) {
#ifdef __CUDA_ARCH__
  const int64_t T = __ldg(reinterpret_cast<const long long*>(&t->exp2[uint32_t(F >> 57)]));
#else
  const int64_t T = t->exp2[uint32_t(F >> 57)];
#endif
  const int64_t f = int64_t((F << 7) ^ (1ull << 63)); /* (F mod 2^-7) - 2^-8, Q71 */
  constexpr int64_t kLn2 = 6393154322601327829ll;     /* ln 2, Q63 */
  const int64_t g2 = mulhi_add(0, f, kLn2) << 1;      /* g, Q71 */
  const int32_t gs = int32_t(g2 >> 32);               /* Q39 */
  constexpr int32_t k720 = int32_t((1ll << 31) / 720), k120 = int32_t((1ll << 31) / 120), k24 = int32_t((1ll << 31) / 24);
  constexpr int64_t k6 = (1ll << 62) / 6, k2 = 1ll << 61;
  const int32_t q5 = k120 + (mulhi_s32(gs, k720) >> 7);
  const int32_t q4 = k24 + (mulhi_s32(gs, q5) >> 7);
  const int64_t q3 = k6 + ((int64_t(gs) * q4) >> 8);
  const int64_t q2 = k2 + (mulhi_add(0, g2, q3) >> 7);
  const int64_t w = mulhi_add(0, g2, q2);      /* g q2, Q69 */
  const int64_t gw = mulhi_add(0, g2, w << 3); /* g^2 q2, Q79 */
  const int64_t em1 = g2 + (gw >> 8);          /* Q71 */
  return T + (mulhi_add(0, T, em1) >> 7);
}

/* the double nearest to S 2^(E - 62) for S in [2^62 - 2^8, 2^63) and a result
 * in the normal range */
P3X_HD double d_from_q62(int64_t S, int E) {
  return d_from_bits((uint64_t(uint32_t(E + 1022)) << 52) + uint64_t(S >> 10) + uint64_t((S >> 9) & 1));
}

/* biased exponent field of a positive double, and its 53-bit significand */
P3X_HD uint32_t d_expo(uint64_t u) { return uint32_t(u >> 52) & 0x7ffu; }
P3X_HD uint64_t d_sig(uint64_t u) { return (u & 0xfffffffffffffull) | 0x10000000000000ull; }
/* x is positive and normal */
P3X_HD bool d_normal_pos(uint64_t u) { return uint32_t(u >> 32) - 0x00100000u < 0x7fe00000u; }

/* log2(x) in Q57 for a positive normal x in [2^-63, 2^63) */
P3X_HD int64_t log2_q57(uint64_t u, const FixTables* t) {
  return (int64_t(int32_t(d_expo(u)) - 1023) << 57) + (log2_sig(d_sig(u) << 11, t) >> 5);
}
/* log2(x) in Q57 with the exponent limited to [-63, 62] */
P3X_HD int64_t log2_q57_clamped(uint64_t u, const FixTables* t) {
  int e = int32_t(d_expo(u)) - 1023;
  e = e < -63 ? -63 : (e > 62 ? 62 : e);
  return (int64_t(e) << 57) + (log2_sig(d_sig(u) << 11, t) >> 5);
}
/* 2^y for y in Q57 */
P3X_HD double exp2_q57(int64_t y, const FixTables* t) {
  return d_from_q62(exp2_sig(uint64_t(y) << 7, t), int(y >> 57));
}

/* cube root of a positive normal x: 2^((e + log2 m) / 3), relative error
 * below 2^-58 before the rounding to a double */
P3X_HD double cbrt_int(double x, const FixTables* t) {
  const uint64_t u = d_bits(x);
  const uint32_t eb = d_expo(u), k = mulhi_u32(eb, 0x55555556u), rem = eb - 3 * k; /* 1023 = 3 * 341 */
  const uint64_t X = (uint64_t(rem) << 62) + uint64_t(log2_sig(d_sig(u) << 11, t));       /* Q62, < 3 */
  const uint64_t F = X + mulhi_u64(X, 0x5555555555555555ull);                        /* X / 3, Q64 */
  return d_from_q62(exp2_sig(F, t), int(k) - 341);
}

/* x^c for a positive normal x in [2^-63, 2^63) and 0 < c < 1 in Q63,
 * relative error below 2^-56 before the rounding to a double */
P3X_HD double pow_int(double x, int64_t c, const FixTables* t) {
  const int64_t y = mulhi_s64(log2_q57(d_bits(x), t), c); /* Q56 */
  return d_from_q62(exp2_sig(uint64_t(y) << 8, t), int(y >> 56));
}

/* the double nearest to V 2^-s */
P3X_HD double d_from_fix(int64_t V, int s) {
  const uint64_t neg = uint64_t(V) & (1ull << 63);
  const uint64_t a = neg ? uint64_t(0) - uint64_t(V) : uint64_t(V);
  const int lz = clz_u64(a);
  const uint64_t n = a << (lz & 63);
  const uint64_t r = (uint64_t(uint32_t(1085 - lz - s)) << 52) + (n >> 11) + ((n >> 10) & 1);
  return V == 0 ? 0.0 : d_from_bits(r | neg);
}

/* Coordinate of a table axis in 64-bit fixed point: the interval [0, n - 1]
 * of a value in Qq already limited to [0, n], and the position in it as a Q63
 * weight (1 as 1 - 2^-63). */
struct FixAxis {
  int i;
  int64_t w;
};
P3X_HD FixAxis fix_axis(int64_t x, int q, int n) {
  FixAxis a;
  a.i = int(x >> q);
  a.i = a.i < n ? a.i : n - 1;
  const uint64_t w = uint64_t(x - (int64_t(a.i) << q)) << (63 - q);
  a.w = int64_t(w >> 63 ? (1ull << 63) - 1 : w);
  return a;
}
P3X_HD int64_t fix_clamp(int64_t x, int64_t lo, int64_t hi) { return x < lo ? lo : (x > hi ? hi : x); }

/* Trilinear interpolation of one ice-table column inside one cell from the
 * cell's eight coefficients c[0..7] in fixed point:
 *   c0 + w1 c1 + w4 (c2 + w1 c3) + w5 (c4 + w1 c5 + w4 (c6 + w1 c7)),
 * each coefficient stored times 2 per weight it is multiplied with (a Q63
 * weight halves the product's high word). */
constexpr int kCellCoefs = 8, kCellCols = 4;
P3X_HD int64_t fix_trilinear(const int64_t c[kCellCoefs], int64_t w1, int64_t w4, int64_t w5) {
  const int64_t e = mulhi_add(c[0], w1, c[1]), d = mulhi_add(c[2], w1, c[3]);
  const int64_t b = mulhi_add(c[4], w1, c[5]), a = mulhi_add(c[6], w1, c[7]);
  return mulhi_add(mulhi_add(e, w4, d), w5, mulhi_add(b, w4, a));
}

/* Position of an ice category in the ice table (lookup_ice,
 * p3/impl/p3_table_ice_impl.hpp:80-138): the size axis
 * (log10(qi / ni) + 18) 4.135985... - 10, the rime axis 3 qm / qi + 1 and the
 * density axis, each limited as the reference limits it, 0-based. */
struct IceCell {
  int cell;
  bool odd; /* an argument is infinite, NaN or (qi / ni) not a positive normal number */
  int64_t w1, w4, w5;
};
constexpr int kCellI = 49, kCellR = 3, kCellD = 4, kIceCells = kCellI * kCellR * kCellD;
/* log2_qn: log2(qi / ni), Q57; ratio: qm / qi in Q60, at most 1; rho52: rime
 * density in Q52, at most 1023 (beyond 900 the axis ends) */
P3X_HD FixAxis ice_size_at(int64_t log2_qn) {
  /* d log2(x) + c of the size axis less one, Q55 */
  constexpr int64_t kd = 5741805296813221454ll; /* 4.135985029041767 log10(2), Q62 */
  constexpr int64_t kc = 2285945404318149440ll;  /* 18 * 4.135985029041767 - 11, Q55 */
  const int64_t x1 = mulhi_s64(log2_qn, kd) + kc;
  return fix_axis(fix_clamp(x1, 0, 49ll << 55), 55, kCellI);
}
P3X_HD IceCell ice_cell_at(int64_t log2_qn, uint64_t ratio, uint64_t rho52) {
  const FixAxis a1 = ice_size_at(log2_qn);
  const FixAxis a4 = fix_axis(int64_t(3 * ratio), 60, kCellR);
  /* (rho - 50) 0.005 up to 650, 3 + (rho - 650) 0.004 above, Q58 */
  const bool low = rho52 <= (650ull << 52);
  const int64_t k = low ? 5902958103587056517ll : 4722366482869645213ll; /* 0.005, 0.004 in Q70 */
  const int64_t x5 = mulhi_add(low ? 0 : (3ll << 58), int64_t(rho52) - (int64_t(low ? 50 : 650) << 52), k);
  const FixAxis a5 = fix_axis(fix_clamp(x5, 0, 4ll << 58), 58, kCellD);
  return IceCell{(a5.i * kCellR + a4.i) * kCellI + a1.i, false, a1.w, a4.w, a5.w};
}
/* The same from doubles.  rhop: 0 or positive; ratio_qm = qm / qi >= 0; qi_ni =
 * qi / ni positive. */
P3X_HD uint64_t rho_q52(double rhop) {
  const uint64_t up = d_bits(rhop);
  const int ep = int(d_expo(up)) - 1023;
  return ep > 9 ? (1023ull << 52) : (ep >= 0 ? d_sig(up) << ep : 0);
}
P3X_HD IceCell ice_cell(double qi_ni, double ratio_qm, double rhop, const FixTables* t) {
  const uint64_t ux = d_bits(qi_ni), ur = d_bits(ratio_qm);
  const int er = 1023 - int(d_expo(ur));
  const uint64_t q60 = er <= 0 ? (1ull << 60) : ((d_sig(ur) << 8) >> (er < 63 ? er : 63));
  IceCell c = ice_cell_at(log2_q57_clamped(ux, t), q60, rho_q52(rhop));
  c.odd = !d_normal_pos(ux) || er == -1024 || d_expo(d_bits(rhop)) == 2047u;
  return c;
}
/* The quotient a / b of two positive normal doubles, unrounded: S 2^(e - 63)
 * with S in [2^62, 2^64). */
struct RawQuotient {
  uint64_t S;
  int e;
};
P3X_HD RawQuotient raw_quotient(double a, double b) {
  const uint64_t ua = d_bits(a), ub = d_bits(b);
  return RawQuotient{sig_quotient(d_sig(ua), d_sig(ub)), int(d_expo(ua)) - int(d_expo(ub))};
}
/* its log2 in Q57, the exponent limited to [-63, 62] */
P3X_HD int64_t log2_of(const RawQuotient& q, const FixTables* t) {
  const int low = int(q.S >> 63) ^ 1;
  int e = q.e - low;
  e = e < -63 ? -63 : (e > 62 ? 62 : e);
  return (int64_t(e) << 57) + (log2_sig(q.S << low, t) >> 5);
}
/* its value in Qn for a value below 2^(63 - n) */
P3X_HD uint64_t fix_of(const RawQuotient& q, int n) {
  const int sh = 63 - n - q.e;
  return q.S >> (sh < 63 ? (sh > 0 ? sh : 0) : 63);
}
/* a rime density m / b in Q52 for ice_cell_at (512 to 1023 comes with e = 10
 * where the quotient of the significands is below one) */
P3X_HD uint64_t rho_q52(const RawQuotient& q) { return q.e > 10 ? (1023ull << 52) : fix_of(q, 52); }

/* value of one column in a cell: c points to its eight coefficients */
P3X_HD int64_t ice_cell_value(const int64_t* c, const IceCell& p) {
  int64_t k[kCellCoefs];
#ifdef __CUDA_ARCH__
#pragma unroll
  for (int j = 0; j < kCellCoefs; j += 2) {
    const longlong2 v = __ldg(reinterpret_cast<const longlong2*>(c + j));
    k[j] = v.x;
    k[j + 1] = v.y;
  }
#else
  for (int j = 0; j < kCellCoefs; ++j) k[j] = c[j];
#endif
  return fix_trilinear(k, p.w1, p.w4, p.w5);
}
/* the same in cell {i of the size axis, 0, 0} with the rime and density weights 0 */
P3X_HD int64_t ice_cell_value_unrimed(const int64_t* c, int64_t w1) {
#ifdef __CUDA_ARCH__
  const longlong2 v = __ldg(reinterpret_cast<const longlong2*>(c));
  return mulhi_add(v.x, w1, v.y);
#else
  return mulhi_add(c[0], w1, c[1]);
#endif
}
/* V 2^-s < 1 for V >= 0 */
P3X_HD bool fix_below_one(int64_t V, int s) { return s >= 0 && (V >> (s < 63 ? s : 63)) == 0; }

/* Rain drop size D = (mu + 1) / lambda with lambda^3 = f n / q, limited to
 * [1e-5, 2e-3] (the reference's limits on lambda, p3_dsd2_impl.hpp:76-126),
 * and its Table3 row coordinate (lookup, p3_table3_impl.hpp:14-64).  In base-2
 * logarithms log2 D = kd - log2(n / q) / 3 with kd = log2(mu + 1) - log2(f) / 3
 * in Q57, so neither lambda nor a division is formed. */
struct RainRow {
  int side;    /* -1: D was below the limits (n too large), 1: above, 0: inside */
  int row;     /* 1-based row of Table3 */
  double frac; /* position between row and row + 1 */
};
P3X_HD RainRow rain_row(int64_t log2_nq, int64_t kd, const FixTables* t) {
  constexpr int64_t kLogMin = -2393701460845809080ll; /* log2(1e-5), Q57 */
  constexpr int64_t kLogMax = -1292105688431629576ll; /* log2(2e-3), Q57 */
  int64_t y = kd - mulhi_s64(log2_nq, 6148914691236517205ll); /* 2^64 / 3 */
  RainRow r;
  r.side = y < kLogMin ? -1 : (y > kLogMax ? 1 : 0);
  y = fix_clamp(y, kLogMin, kLogMax);
  const int64_t D = exp2_sig(uint64_t(y) << 7, t) >> (-9 - int(y >> 57)); /* Q71 */
  const bool fine = D <= 460430732079790408ll;                             /* 195e-6 */
  /* (1e6 D + 5) / 10 below 195 microns, 20 + (1e6 D - 195) / 30 above, Q53 */
  const int64_t c = mulhi_s64(D, fine ? 7036874417766400000ll : 2345624805922133333ll) + (fine ? 1ll << 52 : 27ll << 52);
  r.row = int(c >> 53);
  r.frac = d_from_bits(0x3ff0000000000000ull | ((uint64_t(c) >> 1) & 0xfffffffffffffull)) - 1.0;
  return r;
}

}  // namespace dev
}  // namespace p3x
