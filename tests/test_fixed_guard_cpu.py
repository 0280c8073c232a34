"""The rule that leaves matrices to the FP64 kernels (csrc/zgeev_fixed_guard.cuh), compiled for the host, against
the same rule in numpy, and on the library's own matrix classes (almost none of which it may leave)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tokura_zgeev_batched_gb300 import workloads as wl

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tokura_zgeev_batched_gb300", "csrc")
SOURCE = """
#include <cmath>
#include <cstring>
#include "zgeev_fixed_guard.cuh"
using namespace tzg;
struct OneLane {
  static constexpr int kLanes = 1;
  int rank = 0;
  void sync() const {}
  unsigned long long ior(unsigned long long v) const { return v; }
  int imax(int v) const { return v; }
};
// Column-major n x n complex matrices.
extern "C" void left(const long long* a, int n, int batch, int* out) {
  int scale[128];
  for (int j = 0; j < batch; ++j, a += 2 * n * n) {
    int emax = 0;
    for (int e = 0; e < 2 * n * n; ++e) {
      const int x = (int)(size_of(a[e]) >> 20);
      emax = x > emax ? x : emax;
    }
    const auto size = [&](int r, int c) {
      const unsigned x = size_of(a[2 * (c * n + r)]), y = size_of(a[2 * (c * n + r) + 1]);
      return x > y ? x : y;
    };
    out[j] = emax != 0 && left_to_fp64(OneLane(), n, emax, size, size, scale);  // subnormal ones: not asked
  }
}
"""


@pytest.fixture(scope="module")
def left(tmp_path_factory):
    d = tmp_path_factory.mktemp("guard")
    (d / "guard.cpp").write_text(SOURCE)
    so = str(d / "guard.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "guard.cpp"), "-o", so])
    lib = ctypes.CDLL(so)

    def call(A):
        A = np.ascontiguousarray(np.swapaxes(A, 1, 2), dtype=np.complex128)  # column-major
        out = np.zeros(len(A), dtype=np.int32)
        lib.left(A.ctypes.data_as(ctypes.c_void_p), A.shape[1], len(A), out.ctypes.data_as(ctypes.c_void_p))
        return out.astype(bool)
    return call


NONE = -100000


def exponents(A):
    m = np.maximum(np.abs(A.real), np.abs(A.imag))
    return np.where(m > 0, np.frexp(m)[1] - 1, NONE)


def rule(A):
    e = exponents(A)
    top = e.max((1, 2))[:, None]
    row, column = e.max(2), e.max(1)
    both = np.maximum(row, column)
    return (((row > NONE) & (top - row > 8)) | ((column > NONE) & (top - column > 12)) |
            ((both > NONE) & (top - both > 5))).any(1) | unbalanced(e)


def unbalanced(e):
    """The span of the scales that balance a matrix, in eighths of a binade, all indices at once."""
    n = e.shape[1]
    off = np.where(e > NONE, 8 * e, 8 * NONE)
    off[:, np.arange(n), np.arange(n)] = 8 * NONE
    s = np.zeros(e.shape[:2], dtype=np.int64)
    found = np.zeros(len(e), dtype=bool)
    live = None
    for step in range(16):
        row, column = (off + s[:, None, :]).max(2), (off - s[:, :, None]).max(1)
        d = np.where((row > 4 * NONE) & (column > 4 * NONE), row - column - 2 * s, 0)
        if live is None:
            start = 8 * (10 if n == 2 else max(3, -(-16 // (n - 1))))
            live = (d.max(1) >= start) & (d.min(1) <= -start)
        live = live & (np.abs(d).max(1) >= 4)
        s = s + np.where(live[:, None], np.sign(d) * (np.abs(d) // 2), 0)
        span = s.max(1) - s.min(1)
        found |= live & (span >= 64)
        live = live & ~found & (span >= (32 if step >= 2 else 0))
    return found


def graded(n, seed):
    """Rows, columns, both, and single entries scaled down by all kinds of powers of two, zeros among them."""
    rng = np.random.default_rng(seed)
    A = wl.gaussian(600, n, seed=seed)
    for M in A:
        for _ in range(rng.integers(0, 3)):
            i, s = rng.integers(n), 2.0 ** -float(rng.choice([3, 5, 6, 8, 9, 12, 13, 30, 61, 62, 200, 1000, 1070]))
            kind = rng.integers(4)
            if kind in (0, 2):
                M[i] *= s
            if kind in (1, 2):
                M[:, i] *= s
            if kind == 3:
                M[i] = 0
    A[5] = 0
    A[6] = 2.0 ** -1070 * np.round(4 * A[6])  # subnormal as a whole
    return A


@pytest.mark.parametrize("n", [2, 3, 5, 9, 33])
def test_the_rule(left, n):
    A = graded(n, 6000 + n)
    want = rule(A)
    assert want.any() and not want.all()
    assert np.array_equal(left(A), want)


def scaled(n, seed):
    """D^-1 B D for tridiagonal, Hessenberg and dense B and all kinds of D."""
    rng = np.random.default_rng(seed)
    A = wl.gaussian(400, n, seed=seed)
    for j, M in enumerate(A):
        if j % 3 == 0:
            M *= np.tri(n, n, 1) * np.tri(n, n, 1).T
        elif j % 3 == 1:
            M *= np.tri(n, n, 1).T
        k = float(rng.choice([0, 1, 2, 3, 4, 6, 9])) / (1 if j % 3 == 0 else max(1, n - 1))
        d = 2.0 ** (k * np.arange(n))
        d = d if j % 2 else d[rng.permutation(n)]
        M *= d / d[:, None]
    return A


@pytest.mark.parametrize("n", [2, 3, 5, 9, 33, 64])
def test_the_rule_on_badly_balanced_matrices(left, n):
    A = scaled(n, 6020 + n)
    want = rule(A)
    assert want.any() and not want.all()
    assert np.array_equal(left(A), want)
    # the scales alone
    only = [j for j in range(len(A)) if unbalanced(exponents(A[j:j + 1]))[0]]
    assert len(only) >= 20


@pytest.mark.parametrize("n,k,is_left", [(3, 2, False), (8, 1, False), (64, 1, False), (6, 2, True), (12, 2, True),
                                         (6, 3, True), (12, 3, True), (4, 4, True), (64, 3, True), (4, 8, True)])
def test_scaled_toeplitz_matrices(left, n, k, is_left):
    A = np.diag(np.full(n - 1, 2.0 ** k), 1) + np.diag(np.full(n - 1, 2.0 ** -k), -1) + np.eye(n)
    both = np.stack([A, A.T]).astype(np.complex128)
    assert (left(both) == is_left).all() and (rule(both) == is_left).all()


def test_what_is_below_the_unit_counts(left):
    for s in (-61, -70, -300, -1000):
        A = np.zeros((1, 4, 4), dtype=np.complex128)
        A[0, :2, :2] = [[1, 2], [3, 4]]
        A[0, 2:, 2:] = np.ldexp([[1.0, 2], [3, 4]], s)
        assert left(A).all()
    A[0, 2:, 2:] = 0
    assert not left(A).any()


@pytest.mark.parametrize("n,batch", [(2, 40000), (3, 40000), (4, 40000), (16, 8000), (47, 1003), (64, 500)])
def test_the_usual_classes_are_not_left(left, n, batch):
    """One matrix more in the FP64 launch costs a batch more than it gives."""
    for cls in ("gaussian", "uniform", "vdv", "companion"):
        assert left(wl.GENERATORS[cls](batch, n, seed=6050 + n)).mean() <= 2e-4, cls
