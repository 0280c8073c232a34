// Which matrices are left to the FP64 kernels by their entries' sizes (zgeev_fixed.cuh: fixed point holds an entry
// in absolute terms). The rule reads the input's exponents: what is far below the fixed-point unit is not there any
// more after the conversion, and a row that has become zero looks like one that was.
#pragma once

#include "zgeev_fixed.cuh"

namespace tzg {

// Graded matrices: the small eigenvalues that FP64 gives to its relative precision are held here to an absolute one.
// A matrix is left if the largest entry of a row, of a column, or of the row and the column of one index together is more
// than this many binades below the matrix's largest. Rows and columns of zeros do not count. Worst relative error of an
// eigenvalue, in FP64 and in fixed point, of a few random matrices of orders 4 to 24 against 60 digits:
//   diag(B, 2^-k C)                    k = 4: 5e-15 and 4e-15, k = 6: 4e-15 and 9e-15, k = 10: 8e-15 and 4e-13;
//   D B D, D = diag(1 .. 2^-k)         k = 4: 1e-14 and 5e-15, k = 6: 1e-14 and 6e-14, k = 10: 1e-14 and 1e-11;
//   rows scaled by 1 .. 2^-k           k = 6: 1e-14 and 4e-15, k = 8: 8e-15 and 3e-14, k = 10: 8e-15 and 5e-14;
//   columns scaled by 1 .. 2^-k        k = 10: 3e-13 and 8e-14, k = 12: 7e-13 and 2e-13 (FP64 does not hold these either).
constexpr int kFixedGradedRow = 8;
constexpr int kFixedGradedColumn = 12;
constexpr int kFixedGradedIndex = 5;

// floor(log2 |x|) + 1023 from the bits of |x|, subnormal numbers among them.
TZG_HD int bits_exponent(unsigned long long magnitude) {
  const int e = (int)(magnitude >> 52);
  return e != 0 ? e : 12 - clz64(magnitude);
}
TZG_HD unsigned long long magnitude_bits(long long bits) { return (unsigned long long)bits & 0x7fffffffffffffffull; }

// `top(r, c)`: magnitude_bits of the larger component of an entry; `emax`: the largest exponent field. The lanes of
// `G` take the indices i (row i and column i) in turn; all of them get the answer.
template <class Group, class Top>
TZG_HD bool left_to_fp64(const Group& G, int n, int emax, Top top) {
  bool graded = false;
  for (int i = G.rank; i < n; i += Group::kLanes) {
    unsigned long long row = 0, column = 0;
    for (int k = 0; k < n; ++k) {
      const unsigned long long a = top(i, k), b = top(k, i);
      row = a > row ? a : row;
      column = b > column ? b : column;
    }
    const unsigned long long both = row > column ? row : column;
    graded |= row != 0 && emax - bits_exponent(row) > kFixedGradedRow;
    graded |= column != 0 && emax - bits_exponent(column) > kFixedGradedColumn;
    graded |= both != 0 && emax - bits_exponent(both) > kFixedGradedIndex;
  }
  return G.ior(graded) != 0;
}

}  // namespace tzg
