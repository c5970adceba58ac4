"""The arithmetic of the FP64 Gram's digit products (csrc/dense64.cu k_syrk_digits,
csrc/digits.cuh) restated and checked against exact rationals: a power of two per column and
32-row block, digits, kept diagonals, the blocks' sums in 128-bit integers, one rounding to
FP64, and the guard that gives an output back to FP64 sums.

Per term the digit pairs that are not formed are below 7 * 2^14 * 256^-10 * 2^2.01 of the
product of the two powers of two and the rounding of the entries below 2^-63 of it, together
2^-60.8; 32 terms lose at most 2^-55.8 of a block's unit, and shifting out what is below 2^-88
of the largest powers of two adds 2^-59 of a unit of 2^-29 (smaller ones count as that).  An
output passes the guard if S = sum |x y| is at least 1/96 of the root of the sum of its nb
blocks' squared units (1% for S in FP16): the losses are then below sqrt(nb) 97 (2^-55.8 + 2^-59) S
< sqrt(nb) 2^-49 S, and the rounding is 2^-53 of the result."""
from fractions import Fraction

import numpy as np
import pytest

from test_cpu_digit_rows import digits, to_fixed

BLOCK, GUARD, FRAC = 32, Fraction(1, 96), 18


def exponent(col):
    """The least e with all |x| < 0.9942 2^e (by the mantissa's leading bits); zero columns: low."""
    mx = np.abs(col).max()
    if mx == 0.0:
        return -1022
    m, e = np.frexp(mx)
    return int(e) + (1 if int((2 * m - 1) * (1 << 20)) >= 0xFD000 else 0)


def block_sum(x, y, ex, ey):
    """sum x y of a block over the kept digit pairs, in units of 2^(ex + ey - 70)."""
    dx = [digits(to_fixed(v, 63 - ex)) for v in x]
    dy = [digits(to_fixed(v, 63 - ey)) for v in y]
    S = [sum(a[k] * b[D - k] for a, b in zip(dx, dy) for k in range(D + 1)) for D in range(8)]
    assert max(map(abs, S)) <= 2 ** 22          # exact in the accumulators
    fr = S[6] * 256 + S[7]
    whole = sum(S[D] << (40 - 8 * D) for D in range(6))
    assert abs(whole) < 2 ** 62 and abs(fr) < 2 ** 31
    return (whole << 16) + fr


def int128_double(v, e):
    """v 2^e rounded to FP64 by way of 62 bits and a sticky one."""
    a, s = abs(v), 0
    if a >= 1 << 63:
        s = a.bit_length() - 62
        a = (a >> s) | (1 if a & ((1 << s) - 1) else 0)
    assert a < 1 << 63
    return float((-a if v < 0 else a) * Fraction(2) ** (e + s))


def output(x, y):
    """(value, accepted by the guard, exact value, S) of one output."""
    nb = -(-len(x) // BLOCK)
    cut = [slice(b * BLOCK, (b + 1) * BLOCK) for b in range(nb)]
    ex, ey = [exponent(x[c]) for c in cut], [exponent(y[c]) for c in cut]
    tx, ty = max(ex), max(ey)
    total, size, unit = 0, Fraction(0), Fraction(0)
    for c, a, b in zip(cut, ex, ey):
        d = a - tx + b - ty
        v = block_sum(x[c], y[c], a, b)
        total += v << (d + FRAC) if d >= -FRAC else v >> min(-FRAC - d, 127)
        assert abs(total) < 2 ** 127
        s = sum(abs(Fraction(float(p)) * Fraction(float(q))) for p, q in zip(x[c], y[c])) / Fraction(2) ** (a + b)
        if s > 0:
            u = Fraction(2) ** max(d, -29)
            size += s * Fraction(2) ** d if d >= -60 else 0
            unit += u * u
    exact = sum(Fraction(float(p)) * Fraction(float(q)) for p, q in zip(x, y))
    S = sum(abs(Fraction(float(p)) * Fraction(float(q))) for p, q in zip(x, y))
    return Fraction(int128_double(total, tx + ty - 70 - FRAC)), size * size >= GUARD ** 2 * unit, exact, S


def _inputs(kind, rng, K):
    x, y = rng.standard_normal(K), rng.standard_normal(K)
    x[rng.random(K) < 0.3] = 0.0
    if kind == "tail":
        x, y = x * np.exp(2 * rng.standard_normal(K)), y * np.exp(2 * rng.standard_normal(K))
    if kind.startswith("spike"):
        r = rng.choice(K, 2, replace=False)
        x[r] = 2.0 ** int(kind[5:])
        y[r] = 0.0
    if kind == "disjoint":
        x[::2], y[1::2] = 0.0, 0.0
    if kind == "wide":
        x, y = x * np.exp2(rng.uniform(-60, 0, K)), y * np.exp2(rng.uniform(-60, 0, K))
    return x, y


@pytest.mark.parametrize("kind", ["plain", "tail", "spike8", "spike20", "spike40", "disjoint", "wide"])
def test_accepted_outputs_are_as_good_as_fp64_sums(kind):
    rng = np.random.default_rng(len(kind))
    accepted = 0
    for _ in range(12):
        K = int(rng.integers(40, 400))
        x, y = _inputs(kind, rng, K)
        v, ok, exact, S = output(x, y)
        if not ok:
            continue
        accepted += 1
        nb = -(-K // BLOCK)
        loss = Fraction(int(np.ceil(np.sqrt(nb) * 2 ** 8)), 2 ** 8) * Fraction(2) ** -49 * S
        assert abs(v - exact) <= loss + Fraction(2) ** -53 * (abs(exact) + loss)
    assert accepted == 12 if kind in ("plain", "disjoint") else True
    if kind in ("spike20", "spike40"):
        assert accepted == 0       # the guard sees that S is far below the blocks' units
    if kind == "disjoint":
        assert S == 0 and v == 0


@pytest.mark.parametrize("v", [0, 1, -1, 2 ** 62 - 1, 2 ** 62, -(2 ** 63), 2 ** 63 + 2 ** 9, 2 ** 90 + 2 ** 37, 2 ** 90 + 2 ** 37 + 1,
                               -(2 ** 90 + 3 * 2 ** 37), 2 ** 126 - 1, -(2 ** 127 - 12345)])
def test_rounding_of_128_bit_sums(v):
    assert int128_double(v, -88) == float(v * Fraction(2) ** -88)
