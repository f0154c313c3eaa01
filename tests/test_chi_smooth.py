"""The host predicate that lets P0 take digit operands (chi_smooth): the weights
d / (d^2 - w^2) over the transitions d are positive and within a factor of 64 of
each other for every real shift up to wmax (no GPU)."""
import ctypes as C

import numpy as np
import pytest


def smooth(e, nocc, wmax):
    from quasix_b200 import _native
    f = _native.load()._ZN2qx10chi_smoothEPKdiid
    f.restype = C.c_bool
    e = np.ascontiguousarray(e, dtype=np.float64)
    return f(C.c_void_p(e.ctypes.data), C.c_int(nocc), C.c_int(e.size - nocc), C.c_double(wmax))


@pytest.mark.parametrize("ratio", [2.0, 12.0, 13.0, 40.0, 63.9, 64.1, 500.0])
@pytest.mark.parametrize("frac", [0.0, 0.3, 0.6, 0.85, 0.8999, 0.9001])
def test_bound_is_that_of_the_weights(ratio, frac):
    lo = 0.4
    e = np.array([-0.3 - (ratio - 1.0) * lo, -0.3, -0.3 + lo])
    d = np.linspace(lo, ratio * lo, 2000)
    w = frac * lo
    spread = max(np.ptp(np.log(1 / d)), np.ptp(np.log(d / (d * d - w * w))))
    assert smooth(e, 2, w) == smooth(e, 2, -w) == (frac < 0.9 and spread <= np.log(64.0))


def test_unusable_energies():
    assert not smooth([-1.0, 0.3, 0.2, 1.0], 2, 0.0)
    assert not smooth([-1.0, np.nan, 0.2, 1.0], 2, 0.0)
