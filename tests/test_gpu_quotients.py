"""Quotients by multiplication (apbs_b200/csrc/quotients.cuh) against the division:
div_by to the bit for operands of every exponent, sign and special value, divisors
next to a power of two and of all ones among them; reciprocal to an ulp."""
import ctypes

import numpy as np
import pytest

from apbs_b200.vpmg import lib

pytestmark = pytest.mark.gpu


def _quotients(a, b):
    dp = ctypes.POINTER(ctypes.c_double)
    out = np.zeros((3, a.size))
    assert lib().pmgb_debug_quotients(a.size, a.ctypes.data_as(dp), b.ctypes.data_as(dp),
                                      out.ctypes.data_as(dp)) == 1
    return out


def _operands(rng, n, lo, hi):
    frac = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    edge = rng.integers(0, 4, n)
    frac = np.where(edge == 0, rng.integers(0, 4, n).astype(np.uint64), frac)
    frac = np.where(edge == 1, np.uint64((1 << 52) - 1) - rng.integers(0, 4, n).astype(np.uint64),
                    frac)
    e = rng.integers(lo + 1023, hi + 1024, n).astype(np.uint64)
    sign = rng.integers(0, 2, n).astype(np.uint64)
    return (sign << np.uint64(63) | e << np.uint64(52) | frac).view(np.float64)


@pytest.mark.parametrize("alo,ahi,blo,bhi", [(-3, 3, -3, 3), (-60, 60, -30, 30),
                                             (-1023, 1024, -1023, 1024),
                                             (-1023, -960, -205, 10), (1000, 1024, -10, 205)])
def test_div_by_is_the_division(alo, ahi, blo, bhi):
    rng = np.random.default_rng([ahi + 2000, bhi + 2000])
    n = 1 << 20
    a, b = _operands(rng, n, alo, ahi), _operands(rng, n, blo, bhi)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1.0, -3.0])
    a[:9000], b[9000:18000] = np.tile(special, 1000), np.tile(special, 1000)
    a[18000:18081], b[18000:18081] = np.repeat(special, 9), np.tile(special, 9)
    want, got, _ = _quotients(a, b)
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(want[~nan].view(np.uint64), got[~nan].view(np.uint64))


def test_reciprocal_is_within_an_ulp():
    rng = np.random.default_rng(3)
    b = np.concatenate([_operands(rng, 1 << 20, -8, 8), _operands(rng, 1 << 20, -1000, 1000)])
    want, _, y = _quotients(np.ones_like(b), b)
    assert np.abs(want.view(np.int64) - y.view(np.int64)).max() <= 1
