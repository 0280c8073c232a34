"""The fixed-point building blocks (csrc/zgeev_fixed.cuh) compiled for the host: the rotation
coefficients are unitary to 2^-55, a rotation's outputs are within two units of the exact ones,
and entries up to the stated bounds do not overflow."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tokura_zgeev_batched_gb300", "csrc")
SOURCE = """
#include <cmath>
#include "zgeev_fixed.cuh"
using namespace tzg;
extern "C" void rot(const long long* in, long long* out) {  // x, y | pair (a, b) as V values
  const RotC g = make_rotc(in[0], in[1], in[2]);
  const cfx a = {in[3] + kZero, in[4] + kZero}, b = {in[5] + kZero, in[6] + kZero};
  cfx o, p;
  rotate(make_starts(1), g.cr, g.ci, negated(g.ci), g.s, negated(g.s), a, b, o, p);
  out[0] = value(g.cr); out[1] = value(g.ci); out[2] = value(g.s);
  out[3] = o.x - kZero; out[4] = o.y - kZero; out[5] = p.x - kZero; out[6] = p.y - kZero;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    (d / "rot.cpp").write_text(SOURCE)
    so = str(d / "rot.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "rot.cpp"), "-o", so])
    return ctypes.CDLL(so)


def call(lib, *v):
    i, o = (ctypes.c_longlong * 7)(*v), (ctypes.c_longlong * 7)()
    lib.rot(i, o)
    return list(o)


def check(lib, x, y, a, b):
    cr, ci, s, *got = call(lib, *x, y, *a, *b)
    one = Fraction(1 << 62)
    c2 = (Fraction(cr) ** 2 + Fraction(ci) ** 2 + Fraction(s) ** 2) / one ** 2
    assert abs(c2 - 1) < Fraction(1, 2 ** 55)
    assert max(abs(cr), abs(ci), abs(s)) <= (1 << 62) + (1 << 6)
    exact = [cr * a[0] - ci * a[1] + s * b[0], cr * a[1] + ci * a[0] + s * b[1],
             cr * b[0] + ci * b[1] - s * a[0], cr * b[1] - ci * b[0] - s * a[1]]
    for g, e in zip(got, exact):
        # half a unit of rounding, and three left-out products of halves of at most a unit each
        assert abs(g - Fraction(e) / one) <= Fraction(7, 2)
    return cr, ci, s


def test_random_rotations(lib):
    rng = np.random.default_rng(7)
    for _ in range(3000):
        sh = rng.integers(0, 60, 3)
        v = [int(rng.integers(-2 ** 62 + 1, 2 ** 62)) >> int(t) for t in sh]
        r = [int(t * 0.3 * 2 ** 63) for t in rng.uniform(-1, 1, 4)]
        cr, ci, s = check(lib, (v[0], v[1]), v[2], (r[0], r[1]), (r[2], r[3]))
        n = np.longdouble(v[0]) ** 2 + np.longdouble(v[1]) ** 2 + np.longdouble(v[2]) ** 2
        if n > 0:
            n = np.sqrt(n)
            for c, x in zip((cr, ci, s), v):
                assert abs(np.longdouble(c) / 2 ** 62 - np.longdouble(x) / n) < 2.0 ** -52  # FP64 long double: 2^-53


@pytest.mark.parametrize("v", [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 0, 1), (0, 0, -1), (0, -1, 0), (1, 1, 1),
                               (2 ** 62 - 1, 0, 0), (-2 ** 62 + 1, -2 ** 62 + 1, 2 ** 62 - 1), (2 ** 61, 0, 0),
                               (0, 2 ** 32, 2 ** 31), (-2 ** 31, 2 ** 31 - 1, 2 ** 32 - 1)])
def test_edges(lib, v):
    big = int(0.65 * 2 ** 63)
    for a, b in (((big, 0), (0, 0)), ((0, -big), (0, 0)), ((-big // 2, big // 2), (big // 2, -big // 2)),
                 ((2 ** 31, -2 ** 31), (2 ** 32 - 1, 1)), ((0, 0), (0, 0))):
        cr, ci, s = check(lib, v[:2], v[2], a, b)
    if v[2] == 0:
        assert s == 0  # exactly: what the rotation's second entry holds must not matter
