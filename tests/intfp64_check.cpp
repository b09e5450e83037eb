/* Host check of the integer-arithmetic FP64 operations (p3x_intfp64.cuh is
 * plain integer code on the host too).
 *   check div FAMILY N   disagreements with IEEE division
 *   check FUNC FAMILY N  largest error against extended precision, in units of
 *                        2^-52 of the result (log2: absolute, in 2^-52; ice:
 *                        relative; rain: absolute, of the table coordinate) */
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "p3x_fixtables.hpp"
#include "p3x_intfp64.cuh"

using namespace p3x::dev;

static std::mt19937_64 g(20240);
static double range(int lo, int hi) {
  return d_from_bits((g() & 0x800fffffffffffffull) | (uint64_t(1023 + lo + int(g() % uint64_t(hi - lo + 1))) << 52));
}
static double edge() {
  const uint64_t m = (g() & 1) ? 0xfffffffffffffull - g() % 4 : g() % 4;
  return d_from_bits((uint64_t(1003 + g() % 40) << 52) | m);
}

static long check_div(int family, long n) {
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    double a = 0, b = 1;
    switch (family) {
      case 0: a = range(-300, 300); b = range(-300, 300); break; /* ordinary */
      case 1: a = edge(); b = edge(); break;                     /* significands near 1 and 2 */
      case 2: b = range(-10, 10); a = range(-10, 10) * b; break; /* quotients near a double */
      case 3: a = double(g() % 100000); b = double(1 + g() % 1000); break;
      case 4: a = d_from_bits(g()); b = d_from_bits(g()); break; /* any bits: inf, NaN, subnormal, overflow */
      case 5: a = (g() & 1) ? 0.0 : -0.0; b = range(-300, 300); break;
      case 6: a = range(-1022, -960); b = range(40, 70); break;  /* quotients around the smallest normal */
      case 7: b = range(-3, 3); a = d_from_bits(d_bits(b) + g() % 16); break;
    }
    const double got = ddiv_int(a, b), want = a / b;
    if (d_bits(got) != d_bits(want) && !(std::isnan(got) && std::isnan(want))) ++bad;
  }
  return bad;
}

static long double clampl(long double x, long double lo, long double hi) { return x < lo ? lo : (x > hi ? hi : x); }

/* One ice-table column through the fixed-point cells against lookup_ice and
 * apply_table_ice in extended precision, relative.  Families: 0 inside the
 * axes, 1 at and beyond the ends of each axis and on grid points, 2 rime
 * density next to the axis break at 650. */
static long double check_ice(int family, long n, const FixTables& t) {
  std::vector<double> ice(size_t(p3x::kIceTableSize));
  for (double& v : ice) v = std::exp2(double(g() % 3000) / 1000.0 - 20.0);
  const int cols[kCellCols] = {0, 1, 6, 7};
  std::vector<int64_t> coef;
  std::vector<int32_t> shift;
  p3x::build_ice_cells(ice.data(), cols, coef, shift);
  long double worst = 0;
  for (long i = 0; i < n; ++i) {
    double q_n = std::exp2(-52.0 + double(g() % 42000) / 1000.0), rat = double(g() % 1000001) / 1e6,
           rho = 50.0 + double(g() % 850001) / 1000.0;
    if (family == 1) {
      const double k = double(int(g() % 60) - 4);
      q_n = (g() & 1) ? std::pow(10.0, (k + 10) / 4.135985029041767 - 18) : std::ldexp(1.0, -200 + int(g() % 300));
      rat = double(g() % 7) / 3.0;
      rho = (g() & 1) ? 0.0 : 50.0 * double(g() % 25);
    } else if (family == 2) {
      rho = 650.0 + (double(g() % 5) - 2) * 0x1p-42;
    }
    IceCell c = ice_cell(q_n, rat, rho, &t);
    if (i & 1) { /* from unrounded quotients, as sedimentation forms them */
      const double n = 1.0 + double(g() % 1000) / 7.0, q = q_n * n; /* q_n below: what the doubles give */
      const double b = std::ldexp(1.0, int(g() % 40) - 30); /* rho b is exact */
      const RawQuotient rq = raw_quotient(q, n);
      q_n = q / n;
      if (rat <= 1) c = ice_cell_at(log2_of(rq, &t), rat > 0 ? fix_of(raw_quotient(rat, 1.0), 60) : 0,
                                    rho > 0 ? rho_q52(raw_quotient(rho * b, b)) : 0);
      else c = ice_cell(q_n, rat, rho, &t);
    }
    const long double d1 = clampl((std::log10((long double)q_n) + 18) * (long double)4.135985029041767 - 10, 1, 50);
    const long double d4 = clampl(3 * (long double)rat + 1, 1, 4);
    const long double d5 = clampl(rho <= 650 ? ((long double)rho - 50) * 0.005L + 1 : ((long double)rho - 650) * 0.004L + 4, 1, 5);
    const int i1 = std::min(int(d1), 49) - 1, i4 = std::min(int(d4), 3) - 1, i5 = std::min(int(d5), 4) - 1;
    const long double w1 = d1 - i1 - 1, w4 = d4 - i4 - 1, w5 = d5 - i5 - 1;
    for (int col = 0; col < kCellCols; ++col) {
      long double want = 0;
      for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
          for (int d = 0; d < 2; ++d)
            want += (a ? w5 : 1 - w5) * (b ? w4 : 1 - w4) * (d ? w1 : 1 - w1) *
                    ice[size_t(((i5 + a) * p3x::kRimsize + i4 + b) * p3x::kIsize + i1 + d) * p3x::kIceCols + cols[col]];
      const size_t at = size_t(c.cell) * kCellCols + col;
      const double got = d_from_fix(ice_cell_value(&coef[at * kCellCoefs], c), shift[at]);
      worst = std::fmax(worst, std::fabs(got - want) / want);
    }
  }
  return worst;
}

/* Row and position of the rain table: absolute error of the coordinate.
 * Families: 0 inside the limits, 1 around them, 2 around the break at 195
 * microns. */
static long double check_rain(int family, long n, const FixTables& t) {
  long double worst = 0;
  for (long i = 0; i < n; ++i) {
    const double mu = double(g() % 5) * 0.75;
    const double f = 523.6 * (mu + 3) * (mu + 2) * (mu + 1);
    const int64_t kd = std::llroundl((std::log2((long double)mu + 1) - std::log2((long double)f) / 3) * 0x1p57L);
    long double D = std::exp2(-16.6L + (long double)(g() % 7600) / 1000);
    if (family == 1) D = ((g() & 1) ? 1e-5L : 2e-3L) * (1 + ((long double)(g() % 2001) - 1000) * 1e-12L);
    if (family == 2) D = 195e-6L * (1 + ((long double)(g() % 2001) - 1000) * 1e-12L);
    const double n_q = double(std::pow((mu + 1) / D, 3) / f);
    const RainRow r = rain_row(log2_q57_clamped(d_bits(n_q), &t), kd, &t);
    const long double Dx = clampl((mu + 1) / std::cbrt((long double)f * n_q), 1e-5L, 2e-3L);
    const long double c = Dx <= 195e-6L ? (Dx * 1e6L + 5) / 10 : (Dx * 1e6L - 195) / 30 + 20;
    worst = std::fmax(worst, std::fabs((long double)r.row + r.frac - c));
    if (r.row < 1 || r.row > 80) worst = 1;
  }
  return worst;
}

/* operands: 0 any normal in the range, 1 significands at the table's interval
 * edges and next to powers of two, 2 exact powers of two */
static double operand(int family, int lo, int hi) {
  const double x = std::fabs(range(lo, hi));
  if (family == 0) return x;
  if (family == 2) return std::ldexp(1.0, lo + int(g() % uint64_t(hi - lo + 1)));
  const uint64_t m = ((g() % 129) << 45) + (g() % 5) - 2;
  return d_from_bits((d_bits(x) & ~0xfffffffffffffull) + m);
}

int main(int argc, char** argv) {
  const std::string what = argv[1];
  const int family = std::atoi(argv[2]);
  const long n = std::atol(argv[3]);
  if (what == "div") {
    std::printf("%ld\n", check_div(family, n));
    return 0;
  }
  const FixTables& t = kFixTables;
  if (what == "ice" || what == "rain") {
    std::printf("%.6Le\n", what == "ice" ? check_ice(family, n, t) : check_rain(family, n, t));
    return 0;
  }
  long double worst = 0;
  for (long i = 0; i < n; ++i) {
    long double err = 0;
    if (what == "log2") {
      const double x = operand(family, -62, 61);
      err = std::fabs(std::ldexp(static_cast<long double>(log2_q57(d_bits(x), &t)), -57) - std::log2((long double)x));
    } else if (what == "cbrt") {
      const double x = operand(family, -900, 900);
      const long double want = std::cbrt((long double)x);
      err = std::fabs(cbrt_int(x, &t) - want) / std::ldexp(1.0L, std::ilogb(want));
    } else if (what == "pow") {
      const double x = operand(family, -12, 12);
      const int64_t c = int64_t(std::llround(0.54 * 0x1p63)); /* 0.54 as a double, exact in Q63 */
      const long double want = std::pow((long double)x, (long double)0.54);
      err = std::fabs(pow_int(x, c, &t) - want) / std::ldexp(1.0L, std::ilogb(want));
    } else if (what == "exp2") {
      const int64_t y = int64_t(g()) >> 3; /* (-8, 8) in Q57 */
      const long double want = std::exp2(std::ldexp((long double)y, -57));
      err = std::fabs(exp2_q57(y, &t) - want) / std::ldexp(1.0L, std::ilogb(want));
    } else if (what == "fix") {
      const int sh = int(g() % 64);
      const int64_t V = int64_t(g()) >> sh;
      const int s = int(g() % 200) - 100;
      const long double want = std::ldexp((long double)V, -s);
      const double got = d_from_fix(V, s);
      err = V ? std::fabs(got - want) / std::ldexp(1.0L, std::ilogb(want)) : (got == 0.0 ? 0 : 1e9L);
    }
    worst = std::fmax(worst, err);
  }
  std::printf("%.6Lf\n", worst * 0x1p52L);
  return 0;
}
