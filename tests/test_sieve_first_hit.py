"""CPU: first hits of the sieve's thread-per-prime tier (csrc/dr_kernels.cu) in exact arithmetic.

floor(v/p) as floor((v + 1/2) RN(1/p)) for v up to 2^51, and from it the first byte j of a
segment whose value p divides: every value (byte j holds low + j), or odd values only (low odd,
byte j holds low + 2j)."""
import random
from fractions import Fraction

import pytest

PRIMES = (3, 5, 7, 1021, 4099, 65521, 262139, 1048573, 16777213, 2147483629)


@pytest.mark.parametrize("odd", (False, True))
@pytest.mark.parametrize("p", PRIMES)
def test_first_hit(p, odd):
    rng = random.Random(p)
    ks = [0, 1, 2, 3, (1 << 50) // p] + [int(2 ** rng.uniform(0, 50)) // p for _ in range(200)]
    for low in (k * p + d for k in ks for d in (-2, -1, 0, 1, 2, p // 2, p // 2 + 1)):
        if low < 0 or (odd and low % 2 == 0):
            continue
        v = (low - 1) >> 1 if odd else low
        q = (Fraction(2 * v + 1, 2) * Fraction(1.0 / p)).__floor__() & 0xFFFFFFFF
        r = (v - q * p) & 0xFFFFFFFF
        if odd:
            h = p >> 1
            j = h - r + (p if r > h else 0)
        else:
            j = p - r if r else 0
        assert 0 <= j < p and (low + (2 * j if odd else j)) % p == 0
