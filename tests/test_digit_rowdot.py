"""The integer epilogue of the digit contraction (csrc/digit_rowdot.cuh), run on
the host from its source against exact Python integers.

A row of 64 sums s (|s| < 2^62) is normalised to 62 bits and multiplied with
the integers X of a pair (|X| < 2^55 before their shift); the part of each
product above 2^64 is kept.  Per term that drops less than two units (the floors
of the two middle products) and a quarter (low x low).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quasix_b200", "csrc")

HARNESS = """
#include "digit_rowdot.cuh"
using namespace qx::rowdot;
// Sum over 64 columns in units of 2^64, and the shift of the row.
extern "C" int rowdot64(const int64_t* s, const int64_t* X, int64_t* out) {
  uint32_t top = 0;
  for (int c = 0; c < 64; ++c) top |= top_bits(s[c]);
  const int z = norm_shift(top);
  for (int c0 = 0; c0 < 64; c0 += 16) {
    int64_t acc = 0;
    for (int q = c0; q < c0 + 16; ++q) {
      const Words x = words(X[q] << XSHIFT);
      acc += term(x.lo, x.hi, s[q] << z);
    }
    out[c0 / 16] = acc;
  }
  return z;
}
extern "C" int xshift() { return XSHIFT; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rowdot")
    src = d / "rowdot.cpp"
    src.write_text(HARNESS)
    so = d / "rowdot.so"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fwrapv", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)])
    return ctypes.CDLL(str(so))


def _rowdot(lib, s, X):
    s = np.ascontiguousarray(s, np.int64)
    X = np.ascontiguousarray(X, np.int64)
    out = np.zeros(4, np.int64)
    z = lib.rowdot64(*(a.ctypes.data_as(ctypes.c_void_p) for a in (s, X, out)))
    return int(out.astype(object).sum()), z


def _edges():
    for k in range(33, 63):
        for lead in (2 ** k - 1, 2 ** k - 2 ** (k - 32), 2 ** k - 2 ** (k - 33), 2 ** k - 2 ** (k - 31) - 1, 2 ** (k - 1)):
            yield from (lead, -lead, -lead - 1 if lead < 2 ** 62 - 1 else -lead)


@pytest.mark.parametrize("xtop", [2 ** 54 - 1, int(0.995 * 2 ** 55), -int(0.995 * 2 ** 55), 3])
def test_largest_sums_keep_their_sign(lib, xtop):
    rng = np.random.default_rng(0)
    xs = lib.xshift()
    for lead in _edges():
        s = rng.integers(-abs(lead) // 8 - 1, abs(lead) // 8 + 1, 64)
        X = rng.integers(-2 ** 53, 2 ** 53, 64)
        s[17], X[17] = lead, xtop
        got, z = _rowdot(lib, s, X)
        exact = sum((int(x) << xs) * (int(y) << z) for x, y in zip(X, s))
        assert abs(got * 2 ** 64 - exact) <= 64 * 2.25 * 2 ** 64, (lead, z)


def test_sums_of_sixteen_fit(lib):
    """Every term at its largest, all of one sign."""
    xs = lib.xshift()
    for sx in (1, -1):
        for lead in (2 ** 62 - 1, 2 ** 61, 2 ** 62 - 2 ** 30):
            s = np.full(64, lead)
            X = np.full(64, sx * int(0.996 * 2 ** 55))
            got, z = _rowdot(lib, s, X)
            exact = sum((int(x) << xs) * (int(y) << z) for x, y in zip(X, s))
            assert abs(got * 2 ** 64 - exact) <= 64 * 2.25 * 2 ** 64
