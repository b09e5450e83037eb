/* Ice-table cells of the fixed-point FP64 operations (p3x_intfp64.cuh). */
#ifndef P3X_FIXTABLES_HPP
#define P3X_FIXTABLES_HPP

#include <cstdint>
#include <vector>

#include "p3x_intfp64.cuh"
#include "p3x_internal.hpp"

namespace p3x {

/* Fixed-point coefficients of four ice-table columns for every cell
 * [kIceCells][kCellCols][kCellCoefs] and the power of two of each cell and
 * column [kIceCells][kCellCols]: value = fix_trilinear(...) 2^-shift. */
void build_ice_cells(const double* ice, const int cols[dev::kCellCols], std::vector<int64_t>& coef,
                     std::vector<int32_t>& shift);

/* The host's words of the fixed-point self-test (p3x_fixtest.hpp): kFixTestRows
 * rows of kFixTestWords for these coefficients. */
std::vector<int64_t> fix_test_coefficients();
std::vector<uint64_t> fix_test_words(const std::vector<int64_t>& coef);

}  // namespace p3x

#endif
