/*
 * Values of the fixed-point functions of p3x_intfp64.cuh for the self-test: the
 * host and the device, whose high products are different code and whose tables
 * and loads are their own, have to give the same words.  (What rests on the
 * FP32 reciprocal seed, the divisions, differs between the two and is checked
 * against exact arithmetic instead.)
 */
#ifndef P3X_FIXTEST_HPP
#define P3X_FIXTEST_HPP

#include "p3x_intfp64.cuh"

namespace p3x {

constexpr int kFixTestRows = 1 << 16, kFixTestWords = 27, kFixTestCells = 64;

namespace dev {

struct FixTestHash {
  uint64_t h;
  P3X_HD uint64_t operator()() {
    h += 0x9E3779B97F4A7C15ull;
    uint64_t z = h;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
};

/* a positive normal double with an exponent in [lo, hi]; by `kind` any
 * significand, one at an interval's edge of the tables (or 1), or one below 2 */
P3X_HD uint64_t fix_test_operand(FixTestHash& next, uint64_t kind, int lo, int hi) {
  const uint64_t e = uint64_t(1023 + lo + int(next() % uint64_t(hi - lo + 1))) << 52;
  const uint64_t m = next(), mask = 0xfffffffffffffull;
  if ((kind & 3) == 0) return e | (((m % 128) << 45) + (m >> 32) % 3);
  if ((kind & 3) == 1) return e | (mask - (m % 4));
  return e | (m & mask);
}

/* row i of the test; coef: kFixTestCells cells of kCellCoefs coefficients below 2^60 */
P3X_HD void fix_test_row(uint64_t i, const FixTables* t, const int64_t* coef, uint64_t* out) {
  FixTestHash next{i * 0x9E3779B97F4A7C15ull};
  int n = 0;
  /* the approximate high product, at the ends of its range too */
  const uint64_t ends[4] = {0, ~0ull >> 1, 1ull << 63, ~0ull};
  const uint64_t a = (i & 7) == 1 ? ends[next() & 3] : next(), b = (i & 7) == 2 ? ends[next() & 3] : next();
  out[n++] = uint64_t(mulhi_add(int64_t(next()) >> 2, int64_t(a), int64_t(b)));
  const uint64_t x = fix_test_operand(next, i, -62, 61);
  out[n++] = uint64_t(log2_q57(x, t));
  out[n++] = uint64_t(log2_q57_clamped(fix_test_operand(next, i, -1022, 1023), t));
  out[n++] = d_bits(exp2_q57(int64_t(next()) >> 3, t));
  out[n++] = d_bits(cbrt_int(d_from_bits(fix_test_operand(next, i, -900, 900)), t));
  const double c[3] = {.5, .54, 0.28571};
  out[n++] = d_bits(pow_int(d_from_bits(x), int64_t(c[i % 3] * 9223372036854775808.0), t));
  out[n++] = d_bits(d_from_fix(int64_t(next()) >> (next() & 63), int(next() % 200) - 100));
  /* positions in the ice table, inside the axes and beyond their ends */
  const IceCell p = ice_cell(d_from_bits(fix_test_operand(next, i, i & 8 ? -200 : -52, i & 8 ? 200 : -10)),
                             d_from_bits(fix_test_operand(next, i, -62, 1)),
                             (i & 16) ? double(next() % 1100) : d_from_bits(fix_test_operand(next, i, 5, 10)), t);
  out[n++] = uint64_t(p.cell) | uint64_t(p.odd) << 32;
  out[n++] = uint64_t(p.w1);
  out[n++] = uint64_t(p.w4);
  out[n++] = uint64_t(p.w5);
  const IceCell q = ice_cell_at(int64_t(next() % (40ull << 57)) - (55ll << 57), next() % ((1ull << 60) + 1),
                                next() % (1023ull << 52));
  out[n++] = uint64_t(q.cell);
  out[n++] = uint64_t(q.w1);
  out[n++] = uint64_t(q.w4);
  out[n++] = uint64_t(q.w5);
  /* a column's value in a cell */
  const int64_t* const k = coef + (next() % kFixTestCells) * kCellCoefs;
  const int64_t V = ice_cell_value(k, q), W = ice_cell_value(k, p);
  out[n++] = uint64_t(V);
  out[n++] = uint64_t(W);
  out[n++] = uint64_t(ice_cell_value_unrimed(k, q.w1));
  out[n++] = uint64_t(fix_below_one(V & 0x7fffffffffffffffll, int(next() % 80) - 8));
  /* rain drop sizes, inside and beyond the limits */
  const int64_t nq = (i & 32) ? int64_t(next() % (60ull << 57)) - (20ll << 57) : int64_t(next() % (24ull << 57)) + (8ll << 57);
  const RainRow r = rain_row(nq, -(6ll << 57) + (int64_t(next()) >> 8), t);
  out[n++] = uint64_t(uint32_t(r.row)) | uint64_t(uint32_t(r.side)) << 32;
  out[n++] = d_bits(r.frac);
  /* unrounded quotients of given words */
  RawQuotient u;
  u.S = next() | (1ull << 62);
  u.e = int(next() % 160) - 80;
  out[n++] = uint64_t(log2_of(u, t));
  out[n++] = fix_of(u, 60);
  out[n++] = rho_q52(u);
  out[n++] = rho_q52(d_from_bits(fix_test_operand(next, i, -3, 12)));
  const FixAxis ax = fix_axis(int64_t(next() % (49ull << 55) + (i & 1)), 55, kCellI);
  out[n++] = uint64_t(ax.i);
  out[n++] = uint64_t(ax.w);
}

}  // namespace dev
}  // namespace p3x

#endif
