"""The shortened double-float operations of csrc/df64.cuh, in numpy's FP32 (IEEE,
round to nearest, as the kernels' intrinsics): sums of known order and sums with
a power-of-two weight give the general sum's bits, comparisons the sign of the
exact difference."""
from fractions import Fraction

import numpy as np
import pytest

f32 = np.float32


def two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def add(a, b):
    s, e = two_sum(a[0], b[0])
    return s, e + (a[1] + b[1])


def values(rng, n, lo, hi):
    """DF values with exponents lo..hi, lo parts of a few ulp as products leave them."""
    h = (rng.uniform(1, 2, n) * 2.0 ** rng.integers(lo, hi, n) * rng.choice([-1, 1], n)).astype(f32)
    return h, (h * rng.uniform(-4, 4, n).astype(f32) * f32(2.0 ** -24)).astype(f32)


@pytest.mark.parametrize("span", [0, 1, 12, 40])
def test_ordered_sum_has_the_general_sums_bits(span):
    rng = np.random.default_rng(span)
    a, b = values(rng, 20000, -3, 14), values(rng, 20000, -3 - span, 14 - span)
    swap = np.abs(a[0]) < np.abs(b[0])
    a, b = [np.where(swap, y, x) for x, y in zip(a, b)], [np.where(swap, x, y) for x, y in zip(a, b)]
    s = a[0] + b[0]
    lo = (b[0] - (s - a[0])) + (a[1] + b[1])
    want = add(a, b)
    assert np.array_equal(s, want[0]) and np.array_equal(lo, want[1])


def test_scaled_sum_has_the_general_sums_bits():
    rng = np.random.default_rng(5)
    a, b = values(rng, 20000, -12, 14), values(rng, 20000, -12, 14)
    for w in (f32(1), f32(2)):
        wide = np.float64  # one rounding of an exact product and a sum of 24-bit numbers within 2^28
        fma = lambda x, y: (x.astype(wide) * wide(w) + y.astype(wide)).astype(f32)  # noqa: E731
        s = fma(b[0], a[0])
        bb = s - a[0]
        lo = ((a[0] - (s - bb)) + fma(b[0], -bb)) + fma(b[1], a[1])
        want = add(a, (b[0] * w, b[1] * w))
        assert np.array_equal(s, want[0]) and np.array_equal(lo, want[1])


def test_comparison_has_the_exact_sign():
    rng = np.random.default_rng(9)
    a = values(rng, 3000, -3, 14)
    near = (np.nextafter(a[0], f32(np.inf) * rng.choice([-1, 1], 3000).astype(f32)), a[1] * f32(0.5))
    same = (a[0].copy(), np.nextafter(a[1], f32(0)))
    far = values(rng, 3000, -3, 14)
    for b in (near, same, far, a):
        less = ((a[0] - b[0]) + (a[1] - b[1])) < 0
        exact = [Fraction(float(x)) + Fraction(float(y)) < Fraction(float(u)) + Fraction(float(v))
                 for x, y, u, v in zip(*a, *b)]
        assert np.array_equal(less, exact)
