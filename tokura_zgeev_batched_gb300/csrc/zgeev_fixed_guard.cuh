// Which matrices are left to the FP64 kernels by their entries' sizes (zgeev_fixed.cuh: fixed point holds an entry
// in absolute terms). The rule reads the input's exponents: what is far below the fixed-point unit is not there any
// more after the conversion, and a row that has become zero looks like one that was.
#pragma once

#include "zgeev_fixed.cuh"

namespace tzg {

// A row or column whose largest entry is more than this many binades below the matrix's largest makes the matrix a
// graded one. Rows and columns of zeros do not count.
constexpr int kFixedGradedBits = 12;

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
    graded |= row != 0 && emax - bits_exponent(row) > kFixedGradedBits;
    graded |= column != 0 && emax - bits_exponent(column) > kFixedGradedBits;
  }
  return G.ior(graded) != 0;
}

}  // namespace tzg
