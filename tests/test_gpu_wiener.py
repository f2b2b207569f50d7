"""Wiener weights of the plain Final filters (reciprocal estimate, quotient, one correction by the remainder) against
IEEE division.

Bound: the estimate is within 2^-23 of the reciprocal and the quotient within about 2^-22, so with an exact remainder the
corrected quotient is within 2^-45 before its rounding.  It rounds to the other neighbour only where the true
quotient lies that close to a tie: 2 * 2^-45 of its size out of spacings of at least 2^-24, so at most 2^-20 of random
pairs, by one unit.  The test allows eight times as many."""
import numpy as np
import pytest

import bm3d_b200

pytestmark = pytest.mark.gpu

N = 1 << 22
TINY = float(np.finfo(np.float32).tiny)


def units(w, q):
    return np.abs(w.view(np.int32).astype(np.int64) - q.view(np.int32).astype(np.int64))


def log_uniform(rng, lo, hi):
    return np.exp2(rng.uniform(lo, hi, N)).astype(np.float32)


@pytest.mark.parametrize("r2,sg", [
    ((-30, 12), (-12, 4)),          # pictures in [0, 1]
    ((-102, 100), (-60, 100)),      # everything the correction takes
    ((-149, -90), (-126, -60.01)),  # small variances: divided
    ((-149, 127.9), (-126, -60.01)),
    ((-40, 127.9), (124, 127.9)),   # large divisors: divided
])
def test_weights_round_as_the_division(r2, sg):
    rng = np.random.default_rng(5)
    a, b = log_uniform(rng, *r2), log_uniform(rng, *sg)
    w, q = bm3d_b200.wiener_weights(a, b)
    d = units(w, q)
    assert d.max() <= 1 and np.count_nonzero(d) <= 8 * N / 2 ** 20


def test_weights_of_squares_below_the_exact_remainder():
    """Squares below 2^-102 against ordinary variances: the quotient without its correction.  The estimate is
    off by at most 2^-23, two units, and the product by half a one."""
    rng = np.random.default_rng(6)
    w, q = bm3d_b200.wiener_weights(log_uniform(rng, -149, -102), log_uniform(rng, -60, 60))
    assert units(w, q).max() <= 3


def test_special_values():
    inf, nan = np.float32(np.inf), np.float32(np.nan)
    a = np.array([0, 0, 0, TINY, 1, 3e38, 3e38, inf, nan, 1, 0], np.float32)
    b = np.array([TINY, 1, 3e38, TINY, TINY, TINY, 3e38, 1, 1, inf, inf], np.float32)
    w, q = bm3d_b200.wiener_weights(a, b)
    assert np.array_equal(np.isnan(w), np.isnan(q))
    m = ~np.isnan(q)
    assert np.array_equal(w[m], q[m])
