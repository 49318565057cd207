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
