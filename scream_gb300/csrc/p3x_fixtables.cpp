/*
 * Host side of p3x_intfp64.cuh: the fixed-point ice-table cells, in extended
 * precision.
 */
#include "p3x_fixtables.hpp"

#include <cmath>

#include "p3x_fixtest.hpp"

namespace p3x {

void build_ice_cells(const double* ice, const int cols[dev::kCellCols], std::vector<int64_t>& coef,
                     std::vector<int32_t>& shift) {
  coef.assign(size_t(dev::kIceCells) * dev::kCellCols * dev::kCellCoefs, 0);
  shift.assign(size_t(dev::kIceCells) * dev::kCellCols, 0);
  auto at = [&](int jj, int ii, int i, int c) {
    return static_cast<long double>(ice[size_t((jj * kRimsize + ii) * kIsize + i) * kIceCols + cols[c]]);
  };
  /* the power of two each coefficient is stored with: one per weight */
  static const int kWeights[dev::kCellCoefs] = {0, 1, 1, 2, 1, 2, 2, 3};
  for (int jj = 0; jj < dev::kCellD; ++jj)
    for (int ii = 0; ii < dev::kCellR; ++ii)
      for (int i = 0; i < dev::kCellI; ++i)
        for (int c = 0; c < dev::kCellCols; ++c) {
          long double v[2][2][2];
          for (int a = 0; a < 2; ++a)
            for (int b = 0; b < 2; ++b)
              for (int d = 0; d < 2; ++d) v[a][b][d] = at(jj + a, ii + b, i + d, c);
          long double k[dev::kCellCoefs];
          for (int a = 0; a < 2; ++a)
            for (int b = 0; b < 2; ++b) {
              k[4 * a + 2 * b] = v[a][b][0];
              k[4 * a + 2 * b + 1] = v[a][b][1] - v[a][b][0];
            }
          for (int a = 0; a < 2; ++a)
            for (int d = 0; d < 2; ++d) k[4 * a + 2 + d] -= k[4 * a + d];
          for (int m = 0; m < 4; ++m) k[4 + m] -= k[m];
          long double most = 0;
          for (int m = 0; m < dev::kCellCoefs; ++m)
            most = std::fmax(most, std::fabs(std::ldexp(k[m], kWeights[m])));
          const size_t cell = size_t((jj * dev::kCellR + ii) * dev::kCellI + i) * dev::kCellCols + c;
          /* the largest stored coefficient lies in [2^60, 2^61), so that no
           * partial sum reaches 2^63; a cell of (near) zeros stays zero */
          if (!(most > 0x1p-900L) || !std::isfinite(most)) continue;
          int e = 0;
          std::frexp(most, &e);
          const int s = 61 - e;
          shift[cell] = s;
          for (int m = 0; m < dev::kCellCoefs; ++m)
            coef[cell * dev::kCellCoefs + m] = std::llroundl(std::ldexp(k[m], kWeights[m] + s));
        }
}

std::vector<int64_t> fix_test_coefficients() {
  std::vector<int64_t> coef(size_t(kFixTestCells) * dev::kCellCoefs);
  dev::FixTestHash next{1};
  for (int64_t& c : coef) c = int64_t(next()) >> 4;
  return coef;
}

std::vector<uint64_t> fix_test_words(const std::vector<int64_t>& coef) {
  std::vector<uint64_t> out(size_t(kFixTestRows) * kFixTestWords);
  for (int i = 0; i < kFixTestRows; ++i)
    dev::fix_test_row(uint64_t(i), &dev::kFixTables, coef.data(), &out[size_t(i) * kFixTestWords]);
  return out;
}

}  // namespace p3x
