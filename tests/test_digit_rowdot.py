"""The integer epilogue of the digit contraction (csrc/digit_rowdot.cuh), run on
the host from its source against exact Python integers.

A row of 64 sums s (|s| < 2^62) is normalised to 62 bits and multiplied with
the integers X of a pair (|X| < 2^55); the part of each product above 2^60 is kept.  A term's low x low product drops less than a quarter
of a unit, the sum of 16 rounds twice.
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
// Sum over 64 columns in units of 2^60 times the largest of the columns'
// scales (2^-dn), and the shift of the row.
extern "C" int rowdot64(const int64_t* s, const int* dn, const int64_t* X, int64_t* out) {
  uint64_t top = 0;
  for (int c = 0; c < 64; ++c) top |= top_bits(s[c], dn[c]);
  const int z = norm_shift(top);
  for (int c0 = 0; c0 < 64; c0 += TERMS) {
    Sum acc;
    for (int q = c0; q < c0 + TERMS; ++q) {
      const Words x = x_words(X[q]);
      acc.add(x.lo, x.hi, aligned(s[q], z, dn[q]));
    }
    out[c0 / TERMS] = acc.result();
  }
  return z;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rowdot")
    src = d / "rowdot.cpp"
    src.write_text(HARNESS)
    so = d / "rowdot.so"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fwrapv", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)])
    return ctypes.CDLL(str(so))


def _rowdot(lib, s, X, dn=None):
    dn = np.zeros(64, np.int32) if dn is None else np.ascontiguousarray(dn, np.int32)
    s = np.ascontiguousarray(s, np.int64)
    X = np.ascontiguousarray(X, np.int64)
    out = np.zeros(4, np.int64)
    z = lib.rowdot64(*(a.ctypes.data_as(ctypes.c_void_p) for a in (s, dn, X, out)))
    return int(out.astype(object).sum()), z


def _edges():
    for k in range(34, 63):
        for lead in (2 ** k - 1, 2 ** k - 2 ** (k - 32), 2 ** k - 2 ** (k - 33), 2 ** k - 2 ** (k - 31) - 1, 2 ** (k - 1)):
            yield from (lead, -lead, -lead - 1 if lead < 2 ** 62 - 1 else -lead)


@pytest.mark.parametrize("xtop", [2 ** 54 - 1, int(0.995 * 2 ** 55), -int(0.995 * 2 ** 55), 3])
def test_largest_sums_keep_their_sign(lib, xtop):
    rng = np.random.default_rng(0)
    for lead in _edges():
        s = rng.integers(-abs(lead) // 8 - 1, abs(lead) // 8 + 1, 64)
        X = rng.integers(-2 ** 53, 2 ** 53, 64)
        s[17], X[17] = lead, xtop
        got, z = _rowdot(lib, s, X)
        exact = sum(int(x) * (int(y) << z) for x, y in zip(X, s))
        assert abs(got * 2 ** 60 - exact) <= 64 * (0.25 + 2 * 0.5 / 16) * 2 ** 60, (lead, z)


def test_sums_of_sixteen_fit(lib):
    """Every term at its largest, all of one sign."""
    for sx in (1, -1):
        for lead in (2 ** 62 - 1, 2 ** 61, 2 ** 62 - 2 ** 30):
            s = np.full(64, lead)
            X = np.full(64, sx * int(0.996 * 2 ** 55))
            got, z = _rowdot(lib, s, X)
            exact = sum(int(x) * (int(y) << z) for x, y in zip(X, s))
            assert abs(got * 2 ** 60 - exact) <= 64 * (0.25 + 2 * 0.5 / 16) * 2 ** 60


def test_error_has_no_sign(lib):
    """4000 random rows: eight roundings of each, variance 1 / 12, and 64 low
    products of variance 1 / 144; the mean error stays within six of its
    standard deviations."""
    rng = np.random.default_rng(1)
    err = []
    for _ in range(4000):
        s = rng.integers(-2 ** 61, 2 ** 61, 64)
        X = rng.integers(-2 ** 54, 2 ** 54, 64)
        got, z = _rowdot(lib, s, X)
        exact = sum(int(x) * (int(y) << z) for x, y in zip(X, s))
        err.append((got * 2 ** 60 - exact) / 2 ** 60)
    sd = np.sqrt(8 / 12 + 64 / 144)
    assert np.std(err) < 1.1 * sd
    assert abs(np.mean(err)) < 6 * sd / np.sqrt(len(err))


def test_zero_rows(lib):
    assert _rowdot(lib, np.zeros(64), np.full(64, 5))[0] == 0
    assert _rowdot(lib, np.full(64, 5), np.zeros(64))[0] == 0


@pytest.mark.parametrize("graded", ["sums flat", "sums up", "one small column", "all but one empty"])
def test_columns_of_different_scales(lib, graded):
    """The kept bits are those of the products that matter: the error stays
    within 1e-15 of the root-sum-square of the terms (62 and 55 bits less the
    spread of random words, a factor of a thousand)."""
    rng = np.random.default_rng(2)
    for _ in range(200):
        dn = rng.integers(0, 41, 64)
        if graded == "one small column":
            dn = np.where(np.arange(64) == 9, 38, 0)
        if graded == "all but one empty":  # a zero row of W' next to small ones
            dn = np.where(np.arange(64) == 9, 0, 33)
        s = rng.integers(-2 ** 57, 2 ** 57, 64)
        if graded == "sums up":  # equal products, the largest sums where the scale is smallest
            s >>= 40 - dn
        if graded == "one small column":
            s = np.where(dn > 0, 2 ** 61, s >> 40)
        if graded == "all but one empty":
            s = np.where(dn == 0, 0, s)
        X = rng.integers(-2 ** 54, 2 ** 54, 64)
        got, z = _rowdot(lib, s, X, dn)
        terms = [int(x) * (int(y) << 64 >> int(d)) for x, y, d in zip(X, s, dn)]
        rss = sum(t * t for t in terms) ** 0.5 * 2.0 ** (z - 64)
        assert abs(got * 2 ** 60 - (sum(terms) << z >> 64)) <= 1e-15 * rss
