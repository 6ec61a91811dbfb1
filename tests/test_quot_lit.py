"""The two-part constant divisions of the FP64 path (quot_lit of parity_math.cuh), in exact rational
arithmetic on the CPU: every table entry gives the correctly rounded quotient over quot's range, +0 stays
+0, and -0 keeps its sign except where the low part is negative; there no caller passes a -0."""
from __future__ import annotations

import math
import random
import re
from fractions import Fraction as F
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hermite-teno_gb300" / "csrc"
TABLE = re.search(r"g_lit\[kLitCount\] = \{(.*?)\};", (CSRC / "fp3.cuh").read_text(), re.S).group(1)
ENTRIES = [(int(c), float.fromhex(lo)) for c, lo in
           re.findall(r"1\.0 / (\d+)\.0,\s*(-?0x[0-9a-f.]+p[-+]\d+)", re.sub(r"\s+", " ", TABLE))]


def quotient(a, c, lo):
    """fma(a, hi, fma(a, lo, -0)), each rounded once."""
    hi = 1.0 / c
    t = float(F(a) * F(lo)) if a else a * lo + -0.0
    exact = F(a) * F(hi) + F(t)
    return float(exact) if a else a * hi + t


def test_table():
    assert sorted(c for c, _ in ENTRIES) == [3, 6, 24, 1680, 5040, 6720]
    for c, lo in ENTRIES:
        assert lo == float(F(1, c) - F(1.0 / c))


@pytest.mark.parametrize("c,lo", ENTRIES)
def test_correctly_rounded(c, lo):
    rng = random.Random(c)
    ends = [2.0**-500, math.nextafter(2.0**501, 0.0), 1.0, math.nextafter(1.0, 0.0), float(c)]
    some = [math.ldexp(rng.uniform(1, 2), rng.randint(-500, 500)) for _ in range(20000)]
    near = [float(F(k) * c + d) for k in (1, 3, 2**52 - 1, 2**53 - 1) for d in (-1, 0, 1)]  # about multiples of c
    for a in ends + some + near:
        for x in (a, -a):
            assert quotient(x, c, lo) == float(F(x) / c)
    assert math.copysign(1.0, quotient(0.0, c, lo)) == 1.0
    assert math.copysign(1.0, quotient(-0.0, c, lo)) == (1.0 if lo < 0 else -1.0)


def test_no_negative_zero_where_the_low_part_is_negative():
    text = "".join(p.read_text() for p in CSRC.glob("*.cuh")) + "".join(p.read_text() for p in CSRC.glob("*.cu"))
    for c, lo in ENTRIES:
        calls = re.findall(r"quot_lit\((.*?), %d\.0, " % c, text)
        assert calls
        if lo < 0:
            assert all(x.startswith("abs_(") for x in calls), calls
    assert "Zeros keep their sign" not in text
