"""The arithmetic of the digit-product A rows (csrc/digits.cuh) against exact rationals:
fixed point, signed base-256 digits, the kept diagonals and the packed 64-bit value.

Bound: rounding an entry to 63 bits is 2^-64 of its scale and the dropped diagonals are
below 7 * 2^14 * 256^-10 per term, so a sum of n terms of scaled entries at most 0.48
differs from the exact one by at most n * (2 * 0.48 * 2^-64 + 2^-63.1) plus half of the
packed value's unit."""
from fractions import Fraction

import numpy as np
import pytest

ND, FIX = 8, 63


def to_fixed(x, sh):
    v = Fraction(float(x)) * Fraction(2) ** sh
    s = -1 if v < 0 else 1
    return s * int(abs(v) + Fraction(1, 2))


def digits(X):
    u = X + int("80" * ND, 16)
    assert 0 <= u < 1 << (8 * ND)
    d = [((u >> (8 * (ND - 1 - a))) & 255) - 128 for a in range(ND)]
    assert sum(v * 256 ** (ND - 1 - a) for a, v in enumerate(d)) == X
    return d


def up_bits(total):
    e = 0
    while 2 ** e <= total:
        e += 1
    return max(-40, min(8, 9 - e))


def packed(S, up):
    """acc_value: the eight diagonal sums to units of 2^-(56 + up)."""
    v = sum(S[D] << (40 - 8 * D) for D in range(6))
    fr = S[6] * 256 + S[7]
    if up >= 0:
        return (v << up) + (((fr >> (15 - up)) + 1) >> 1)
    return (v + (fr >> 16) + (1 << (-up - 1))) >> -up


def test_rounding_of_coarse_units_is_unbiased():
    """Many packed values of a unit above 2^-56 add up without drift."""
    rng = np.random.default_rng(5)
    S = rng.integers(-(1 << 21), 1 << 21, size=(4000, 8))
    up = -6
    exact = sum(sum(int(s[D]) * 256 ** (7 - D) for D in range(8)) for s in S)       # units of 2^-72
    got = sum(packed([int(v) for v in s], up) for s in S)
    assert abs(got - Fraction(exact, 2 ** (16 - up))) <= 4 * np.sqrt(4000 / 12)


@pytest.mark.parametrize("n,span", [(1, 0), (3, 4), (16, 12), (32, 40)])
def test_products_of_scaled_entries(n, span):
    rng = np.random.default_rng(n)
    for _ in range(20):
        mag = np.exp2(-rng.uniform(0, span, n)) if span else np.ones(n)
        a = rng.uniform(-0.95, 0.95, n) * mag           # rows: the cluster's magnitude
        b = rng.uniform(-0.95, 0.95, n)                 # columns: at most one
        X, Y = [to_fixed(v, FIX) for v in a], [to_fixed(v, FIX) for v in b]
        dx, dy = [digits(v) for v in X], [digits(v) for v in Y]
        S = [sum(dx[c][k] * dy[c][D - k] for c in range(n) for k in range(D + 1)) for D in range(ND)]
        assert max(map(abs, S)) <= 2 ** 22              # exact in the accumulators
        up = up_bits(1.01 * mag.sum())
        V = packed(S, up)
        assert abs(V) < 2 ** 63
        got = Fraction(V) / Fraction(2) ** (56 + up)
        want = sum(Fraction(float(p)) * Fraction(float(q)) for p, q in zip(a, b)) / 4
        bound = n * (2 * Fraction(48, 100) / 2 ** 64 + Fraction(2) ** -63 * Fraction(94, 100)) + Fraction(1, 2 ** (57 + up))
        if up < 0:
            bound += Fraction(1, 2 ** (56 + up))
        assert abs(got - want) <= bound


def test_extreme_digits_fit():
    """The largest magnitudes the scaling allows (0.957 of 2^63) and the accumulators' range."""
    m = int(0.957 * 2 ** 63)
    for X in (m, -m, 0, 1, -1, 2 ** 62, -(2 ** 62)):
        digits(X)
    assert 32 * 8 * 128 * 128 == 2 ** 22
    # columns of a Gram are scaled by their own exponent: entries up to (1 + 0xfd000 / 2^20) / 2
    top = int((1 + Fraction(0xFD000, 1 << 20)) / 2 * 2 ** 63)
    for X in (top - 1, -(top - 1)):
        d = digits(X)
        assert -128 <= min(d) and max(d) <= 127
