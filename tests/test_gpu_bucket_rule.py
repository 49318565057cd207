"""GPU: tables on both sides of the size from which squares are bucketed, which depends on the
threads of a CTA: the same table whatever the shape."""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu

# the prime after the last one that goes unbucketed, per threads of a CTA
NEXT = {128: 20399, 256: 22961, 512: 28183, 1024: 38891}


def test_primes_of_the_rule():
    sieve = bytearray([1]) * 40000
    primes = []
    for p in range(2, 40000):
        if sieve[p]:
            primes.append(p)
            sieve[p * p::p] = bytes(len(sieve[p * p::p]))
    assert {b: primes[2048 + 2 * b] for b in NEXT} == NEXT


@pytest.mark.parametrize("block", sorted(NEXT))
def test_same_table(engine, block):
    q = NEXT[block] ** 2
    for u in (q - 1, q, q + 12345):
        engine.table_build(u, u // 5, 10**6, dr_b200.Params(segment_log2=15, block_threads=block))
        got = engine.table_checksums()
        engine.table_build(u, u // 5, 10**6, dr_b200.Params(segment_log2=17, block_threads=640))
        assert got == engine.table_checksums(), u
