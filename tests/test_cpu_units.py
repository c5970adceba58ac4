"""The unit of packed digit products (csrc/units.h) for any number of terms.

A group of n terms of the largest magnitude has outputs up to n * terms * 0.2481 in units of
2^-(56 + up) (csrc/digits.cuh), so up must leave them below 2^63 for every n -- 2^16 shares
of 65,537 already pass 32 bits -- and not be coarser than that asks for by more than the
power of two it rounds to and the allowance of one share's last bit."""
import os
import subprocess
from fractions import Fraction

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("units") / "units_check")
    subprocess.run(["g++", "-O1", "-std=c++17", os.path.join(HERE, "native", "units_check.cpp"), "-o", out], check=True)
    return out


CASES = [(n, t) for n in (1, 2, 15, 16, 1 << 15, (1 << 16) - 2, (1 << 16) - 1, 1 << 16, (1 << 16) + 1, 1 << 18, 1 << 24,
                          (1 << 31) - 1) for t in (1, 2, 12, 24, 48)]


def test_outputs_fit_63_bits(program):
    args = [str(v) for c in CASES for v in c]
    lines = subprocess.run([program] + args, check=True, capture_output=True, text=True).stdout.split("\n")
    for (n, t), line in zip(CASES, lines):
        up = int(line)
        largest = Fraction(n * t) * Fraction(2481, 10000) * Fraction(2) ** (56 + up)
        assert largest < 2 ** 63, (n, t, up)
        assert up in (8, -40) or largest > Fraction(2) ** 60, (n, t, up)
    assert lines[len(CASES)] == f"{65536 // 8 + 1} 2 2"
