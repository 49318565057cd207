"""CPU: the tile kernel's S2 quotients below y = 2^48, in exact arithmetic.

There it uses the tabulated reciprocals as they are, RN(1/j) with mu(j) in the two low mantissa
bits (up to 3.5 ulp off), and RN(r / 12) for the quotients by 12 j: floor((y + 1/2) r) is still
floor(y / j).  At the y that decide it: multiples and their neighbours, up to the limit."""
import random
import struct
from fractions import Fraction

import pytest

LIMIT = 1 << 48


def with_low_bits(x, bits):
    return struct.unpack("<d", struct.pack("<Q", (struct.unpack("<Q", struct.pack("<d", x))[0] & ~3) | bits))[0]


@pytest.mark.parametrize("seed", range(4))
def test_floor_of_product(seed):
    rng = random.Random(4000 + seed)
    for _ in range(1500):
        j = max(1, int(2 ** rng.uniform(0, 31)))
        for bits in (0, 1, 3):
            r = with_low_bits(1.0 / j, bits)
            for n, rn in ((j, r), (12 * j, r * (1.0 / 12.0))):
                top = LIMIT // n
                qs = {1, top, top - 1, max(1, top // 2), int(2 ** rng.uniform(0, max(0.0, top.bit_length() - 1)))}
                for y in [q * n + d for q in qs for d in (-1, 0, 1, n - 1)] + [LIMIT - 1]:
                    if 1 <= y < LIMIT:
                        assert (Fraction(2 * y + 1, 2) * Fraction(rn)).__floor__() == y // n, (n, y)
