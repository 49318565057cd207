"""CPU: the tile kernel's one-instruction quotient (csrc/dr_tiles.cu) in exact arithmetic.

For y < 2^51 and a reciprocal r of n with relative error at most 2^-53 (1 + 2^-40),
floor((y + 1/2) * r) = floor(y / n), so an FMA rounded down onto integers near 2^52 is the
quotient itself.  Checked with rationals at the y that decide it -- multiples of n and
their neighbours, up to the limit -- for the tabulated RN(1/n) (S1), for the reciprocals
that carry mu(j) in their two low mantissa bits after the Newton step that restores them
(S2), and for 1/(12 j) after its own Newton step.
"""
import random
import struct
from fractions import Fraction

import pytest

MAX_Y = 1 << 51


def fma(a, b, c):
    """RN(a*b + c): float(Fraction) rounds correctly."""
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def with_low_bits(x, bits):
    return struct.unpack("<d", struct.pack("<Q", (struct.unpack("<Q", struct.pack("<d", x))[0] & ~3) | bits))[0]


def newton(n, x):
    return fma(x, fma(-float(n), x, 1.0), x)


def check(n, r, ys):
    for y in ys:
        if 1 <= y < MAX_Y:
            got = (Fraction(2 * y + 1, 2) * Fraction(r)).__floor__()
            assert got == y // n, (n, y)


@pytest.mark.parametrize("seed", range(4))
def test_floor_of_product(seed):
    rng = random.Random(1000 + seed)
    for _ in range(1500):
        n = max(1, int(2 ** rng.uniform(0, 31)))
        top = MAX_Y // n
        qs = {1, top - 1, top, max(1, top // 2), max(1, int(2 ** rng.uniform(0, max(0.0, top.bit_length() - 1))))}
        ys = [q * n + d for q in qs for d in (-1, 0, 1, n - 1)] + [MAX_Y - 1]
        check(n, 1.0 / n, ys)
        for bits in (0, 1, 3):
            check(n, newton(n, with_low_bits(1.0 / n, bits)), ys)
        if n < (1 << 31) // 12:
            r = newton(n, with_low_bits(1.0 / n, rng.choice((0, 1, 3))))
            q12 = r * (1.0 / 12.0)
            r12 = fma(q12, fma(-12.0 * n, q12, 1.0), q12)
            check(12 * n, r12, [12 * y + e for y in ys for e in (-1, 0, 11)])
