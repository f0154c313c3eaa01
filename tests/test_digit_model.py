"""Error model of the digit products behind the FP64 contractions on the
integer tensor pipe (csrc/k_digits.cu), restated in numpy with exact integers
(no GPU).

A row is held as integers X = rint(x 2^(55 - e)), 2^e above its largest entry
by 0.8 % at least, in seven balanced base-256 digits d_i in [-128, 127],
X = sum_i d_i 256^(6 - i).  Of a product of two rows the digit products of
i + j <= 6 are kept.
"""
from fractions import Fraction

import numpy as np
import pytest

BIAS = 0x80808080808080


def _integers(x):
    m, e = np.frexp(np.abs(x).max())
    if m >= 0.9921875:  # the top digit's margin
        e += 1
    return np.rint(np.ldexp(x, 55 - int(e))).astype(np.int64), int(e)


def _digits(X):
    z = (X + np.int64(BIAS)) ^ np.int64(BIAS)
    return [((z >> (8 * (6 - i))) & 255).astype(np.uint8).view(np.int8).astype(np.int64) for i in range(7)]


@pytest.mark.parametrize("lead", [1.0, 0.9921874, 0.9921876, 0.99999999, -1.0, -0.9999])
def test_digits_represent_the_integers(lead):
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, 4000) * np.abs(lead)
    x[0] = lead
    X, e = _integers(x)
    d = _digits(X)
    assert all(-128 <= v.min() and v.max() <= 127 for v in d)
    assert np.array_equal(sum(v << (8 * (6 - i)) for i, v in enumerate(d)), X)
    assert np.abs(np.ldexp(X.astype(float), e - 55) - x).max() <= 2.0 ** (e - 56)


@pytest.mark.parametrize("K,spread", [(64, 0), (1000, 0), (10400, 0), (10400, 3)])
def test_product_error(K, spread):
    """The kept products differ from the exact sum by the two roundings
    (2^-56 of each row's bound per entry) and the dropped digit products
    (at most 6 * 2^14 * 256^-7 (1 + 2^-7) per entry in units of 2^-14 of the bounds)."""
    rng = np.random.default_rng(K)
    a = rng.normal(size=K)
    b = rng.normal(size=K) * 10.0 ** (-spread * rng.uniform(size=K))
    (A, ea), (B, eb) = _integers(a), _integers(b)
    da, db = _digits(A), _digits(B)
    D = [int(sum((da[i] * db[t - i]).sum() for i in range(t + 1))) for t in range(7)]
    assert all(abs(v) < 2 ** 31 for v in D)
    got = sum(Fraction(v, 256 ** t) for t, v in enumerate(D)) * Fraction(2) ** (ea + eb - 14)
    exact = sum(Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b))
    bound = float(np.abs(a).sum()) * 2.0 ** (eb - 56) + float(np.abs(b).sum()) * 2.0 ** (ea - 56)
    bound = bound * 1.01 + K * 6 * 2.0 ** -56 * 1.01 * 2.0 ** (ea + eb)
    assert abs(float(got - exact)) <= bound
    # Random digits: far below the worst case, about an FP64 sum's own error.
    rms = float(np.sqrt((a * a * b * b).sum()))
    assert abs(float(got - exact)) <= 64 * 2.0 ** -53 * rms


def test_accumulators_stay_in_32_bits():
    """Seven products of magnitude 2^14 per value of K, K up to 16384."""
    assert 7 * 2 ** 14 * 16384 < 2 ** 31
