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

// Badly balanced matrices, D^-1 B D: their eigenvalues are as ill-conditioned normwise as D is, but FP64 keeps those of
// banded and Hessenberg ones all the same, having no absolute unit. A matrix is left if the scales that balance it (the
// largest entries beside the diagonal of row i and column i alike) span this many binades. Errors over the norm, FP64 and
// fixed point, tridiagonal 2^k, 1, 2^-k: k = 1, n = 24 7e-12 and 1e-12; k = 2, n = 12 9e-14 and 1e-13, n = 24 7e-9 and
// 1e-6; k = 3, n = 3 4e-17 and 0, n = 6 4e-16 and 2e-15, n = 12 1e-13 and 2e-10; k = 10, n = 4 1e-18 and 1e-10. Relative
// errors of dense ones, D = 1 .. 2^k: k = 6 1e-14 and 2e-14, k = 8 2e-14 and 3e-13. The scales are found in steps, all
// indices at once, in parts of a binade; those of the matrices above span 4 binades in the third step, or never 8, and 8 in
// the 13th at the latest. The search starts when one index's row and another's column are larger by three binades, of small
// orders by 16 / (n - 1), without which a chain of n indices does not span 8 (order 2: by 10, where two entries' digits
// begin to differ, 9e-15 against 5e-16 at 2^12): in hardly any Gaussian matrix, 1 to 11 % of V diag V^-1 ones (with three at all orders: 4,000,000 Gaussian matrices of order 2 1.86 -> 2.16 ms, 2,000,000 V diag V^-1 of
// order 3 2.79 -> 2.89; so 1.91 and 2.81).
constexpr int kFixedUnbalancedBits = 8;
TZG_HD int balance_start(int n) { return n > 6 ? 3 : n == 2 ? 10 : (2 * kFixedUnbalancedBits + n - 2) / (n - 1); }
constexpr int kBalanceParts = 8;
constexpr int kBalanceSteps = 16;

// The size of a number, from its bits: the high word of |x|, with a bit for what is below it (subnormal numbers count,
// if only as far below all others). Then floor(log2 |x|) + 1023 of a size that is not 0.
TZG_HD unsigned size_of(long long bits) {
  return ((unsigned)(bits >> 32) & 0x7fffffffu) | ((unsigned)bits != 0 ? 1u : 0u);
}
TZG_HD int size_exponent(unsigned size) {
  const int e = (int)(size >> 20);
  return e != 0 ? e : 12 - clz32(size);
}

// `top(r, c)`: the larger component's size of an entry; `first(r, c)`: the same, called once for each entry before any
// top (so that a caller can do more with it); `emax`: the largest exponent field; `scale`: 2n words that the lanes of `G`
// share. The lanes take the indices i (row i and column i) in turn; all get the answer.
template <class Group, class First, class Top>
TZG_HD bool left_to_fp64(const Group& G, int n, int emax, First first, Top top, int* scale) {
  bool graded = false, up = false, down = false;
  const int start = balance_start(n);
  for (int i = G.rank; i < n; i += Group::kLanes) {
    unsigned row = 0, column = 0, diagonal = 0;
    for (int k = 0; k < n; ++k) {
      const unsigned b = first(k, i);
      if (k == i)
        diagonal = b;
      else
        column = b > column ? b : column;
    }
    for (int k = 0; k < n; ++k) {
      const unsigned a = k != i ? top(i, k) : 0u;
      row = a > row ? a : row;
    }
    if (row != 0 && column != 0) {
      const int d = size_exponent(row) - size_exponent(column);
      up |= d >= start;
      down |= d <= -start;
    }
    row = diagonal > row ? diagonal : row;
    column = diagonal > column ? diagonal : column;
    const unsigned both = row > column ? row : column;
    graded |= row != 0 && emax - size_exponent(row) > kFixedGradedRow;
    graded |= column != 0 && emax - size_exponent(column) > kFixedGradedColumn;
    graded |= both != 0 && emax - size_exponent(both) > kFixedGradedIndex;
  }
  const unsigned long long found = G.ior((graded ? 1u : 0u) | (up ? 2u : 0u) | (down ? 4u : 0u));
  if (found & 1) return true;
  if (found != 6) return false;
  constexpr int kNone = -(1 << 28), kBias = 1 << 24;  // scales stay far below the bias
  int *now = scale, *next = scale + n;
  for (int i = G.rank; i < n; i += Group::kLanes) now[i] = 0;
  for (int step = 0; step < kBalanceSteps; ++step) {
    G.sync();
    int low = kBias, high = -kBias;
    bool moving = false;
    for (int i = G.rank; i < n; i += Group::kLanes) {
      int row = kNone, column = kNone;
      for (int k = 0; k < n; ++k) {
        if (k == i) continue;
        const unsigned a = top(i, k), b = top(k, i);
        const int r = kBalanceParts * size_exponent(a) + now[k], c = kBalanceParts * size_exponent(b) - now[k];
        if (a != 0 && r > row) row = r;
        if (b != 0 && c > column) column = c;
      }
      const int d = row > kNone && column > kNone ? row - column - 2 * now[i] : 0;
      moving |= d >= kBalanceParts / 2 || d <= -kBalanceParts / 2;
      const int v = now[i] + d / 2;
      next[i] = v;
      low = v < low ? v : low;
      high = v > high ? v : high;
    }
    if (!G.ior(moving)) return false;
    const int span = G.imax(high + kBias) + G.imax(kBias - low) - 2 * kBias;
    if (span >= kFixedUnbalancedBits * kBalanceParts) return true;
    if (step >= 2 && span < kFixedUnbalancedBits / 2 * kBalanceParts) return false;
    int* const t = now;
    now = next;
    next = t;
  }
  return false;
}

}  // namespace tzg
