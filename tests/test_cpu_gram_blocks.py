"""The arithmetic of the FP64 Gram's digit products (csrc/dense64.cu k_syrk_digits,
csrc/digits.cuh) restated and checked against exact rationals: a power of two per column and
64-row block, digits, kept diagonals, the integer sums of a block, one rounding to FP64 per
block, and the guard that gives an output back to FP64 sums.

Per term the digit pairs that are not formed are below 7 * 2^14 * 256^-10 * 2^2.01 of the
product of the two powers of two and the rounding of the entries below 2^-63 of it, together
2^-60.8; 64 terms lose at most 2^-54.8.  An output passes the guard if S = sum |x y| is at least
1/64 of the root of the sum of its nb blocks' squared units (1% for S in FP16): the blocks'
losses are then below sqrt(nb) 64.7 * 2^-54.8 S, and each block's rounding and addition below
2^-52 (S + loss)."""
from fractions import Fraction

import numpy as np
import pytest

from test_cpu_digit_rows import digits, to_fixed

BLOCK, GUARD = 64, Fraction(1, 64)


def exponent(col):
    """The least e with all |x| < 0.9942 2^e (by the mantissa's leading bits); zero columns: low."""
    mx = np.abs(col).max()
    if mx == 0.0:
        return -1022
    m, e = np.frexp(mx)
    return int(e) + (1 if int((2 * m - 1) * (1 << 20)) >= 0xFD000 else 0)


def block_sum(x, y, ex, ey):
    """sum x y of a block over the kept digit pairs, rounded to FP64 in units of 2^(ex + ey)."""
    dx = [digits(to_fixed(v, 63 - ex)) for v in x]
    dy = [digits(to_fixed(v, 63 - ey)) for v in y]
    S = [sum(a[k] * b[D - k] for a, b in zip(dx, dy) for k in range(D + 1)) for D in range(8)]
    whole, part = 0, 0
    for lo in range(0, len(x), 32):   # collect(): 32 rows at a time, exact in the accumulators
        s32 = [sum(a[k] * b[D - k] for a, b in zip(dx[lo:lo + 32], dy[lo:lo + 32]) for k in range(D + 1)) for D in range(8)]
        assert max(map(abs, s32)) <= 2 ** 22
        fr = s32[6] * 256 + s32[7]
        whole += sum(s32[D] << (40 - 8 * D) for D in range(6)) + (fr >> 16)
        part += fr & 0xFFFF
    assert whole * 65536 + part == sum(S[D] << (56 - 8 * D) for D in range(8))
    whole += part >> 16
    assert abs(whole) < 2 ** 62
    sh = min(16, max(64 - abs(whole).bit_length() - 2, 0))
    v = (whole << sh) + ((part & 0xFFFF) >> (16 - sh))
    assert abs(v) < 2 ** 63
    return Fraction(float(v)) * Fraction(2) ** (2 - 56 - sh)


def output(x, y):
    """(value, accepted by the guard, exact value, S) of one output."""
    nb = -(-len(x) // BLOCK)
    cut = [slice(b * BLOCK, (b + 1) * BLOCK) for b in range(nb)]
    ex, ey = [exponent(x[c]) for c in cut], [exponent(y[c]) for c in cut]
    tx, ty = max(ex), max(ey)
    total, size, unit = 0.0, Fraction(0), Fraction(0)
    for c, a, b in zip(cut, ex, ey):
        d = a - tx + b - ty
        total = total + float(block_sum(x[c], y[c], a, b) * Fraction(2) ** d)
        s = sum(abs(Fraction(float(p)) * Fraction(float(q))) for p, q in zip(x[c], y[c])) / Fraction(2) ** (a + b)
        if s > 0:
            u = Fraction(2) ** max(d, -60)
            size += s * u if d >= -60 else 0
            unit += u * u
    exact = sum(Fraction(float(p)) * Fraction(float(q)) for p, q in zip(x, y))
    S = sum(abs(Fraction(float(p)) * Fraction(float(q))) for p, q in zip(x, y))
    return Fraction(total) * Fraction(2) ** (tx + ty), size * size >= GUARD ** 2 * unit, exact, S


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
        loss = Fraction(int(np.ceil(np.sqrt(nb) * 64.7 * 2 ** 8)), 2 ** 8) * Fraction(2 ** -54.8) * S
        assert abs(v - exact) <= loss + nb * Fraction(2) ** -52 * (S + loss)
    assert accepted == 12 if kind in ("plain", "disjoint") else True
    if kind in ("spike20", "spike40"):
        assert accepted == 0       # the guard sees that S is far below the blocks' units
    if kind == "disjoint":
        assert S == 0 and v == 0
