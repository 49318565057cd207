"""GPU: the statistics of a replayed batch are those of the batch, whatever ran in between."""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu


def test_no_bands_of_an_earlier_call():
    xs = [10**9 + k for k in range(8)]
    X = 10**13
    p = dr_b200.default_params(X, dr_b200.POLICY_COMPRESSED)
    with dr_b200.Engine(0) as e:
        e.set_resident_limit(42000000, 10**7)
        e.mertens(X, p)  # the larger buffers first: the second streamed call grows none
        out = e.mertens_batch(xs)[0]
        assert e.mertens(X, p).stats.bands > 0
        again, st = e.mertens_batch(xs)
        assert again == out
        assert (st.bands, st.band_table_ms, st.band_sums_ms) == (0, 0.0, 0.0)


@pytest.mark.parametrize("X,n", [(10**9, 8), (10**15, 3)])  # without and with window work
def test_host_bytes(X, n):
    xs = [X + 1000 * k for k in range(n)]
    p = [dr_b200.default_params(X + 10**6, dr_b200.POLICY_COMPRESSED)] * n
    with dr_b200.Engine(0) as e:
        out, first = e.mertens_batch(xs, p)
        e.mertens(10**6)  # other primes, other staging
        again, st = e.mertens_batch(xs, p)
        assert again == out
        assert (st.h2d_bytes, st.d2h_bytes) == (first.h2d_bytes, first.d2h_bytes)


def test_many_kept_batches():
    """More batches than graphs are kept, of lengths that do and do not fit the staging of the
    one that makes room; each replayed twice, with the others and single queries in between."""
    p = dr_b200.default_params(10**15, dr_b200.POLICY_COMPRESSED)
    batches = [[10**9 + k] * n for k, n in enumerate((3, 200, 5, 40))] + [[10**15 + k] * 3 for k in range(4)]
    with dr_b200.Engine(0) as e:
        want = [[e.mertens(x, p if x > 10**14 else None).M for x in xs] for xs in batches]
        for _ in range(2):
            for xs, w in zip(batches, want):
                ps = [p] * len(xs) if xs[0] > 10**14 else None
                for _ in range(2):
                    assert e.mertens_batch(xs, ps)[0] == w
                assert e.mertens(10**10).M == -33722
