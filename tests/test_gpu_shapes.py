"""GPU: the sieve shape a table takes when the caller names none.

Small tables run 256-thread CTAs on short segments and leave their squares unbucketed.  The
table is the same for every shape, so the default's checksums equal those of 2^18-value
segments and 1024 threads, at the sizes where the rule or the bucket switch steps and for
dense cutoffs inside a segment and on none; a streamed table keeps one shape for its
resident part and its bands.
"""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu

STEPS = [700 << k for k in range(12, 17)]


@pytest.mark.parametrize("u", [1, 63, 4096, 4097, 10**6 + 3, STEPS[1] * 7 // 5 - 1, STEPS[1] * 7 // 5 + 1,
                               STEPS[4] * 7 // 5 + 1, 149999999, 150000000, 38873 * 38873 + 5, 38891 * 38891 + 5])
def test_default_shape_table(engine, u):
    for dense in {u, u // 3, u // 3 // 64 * 64, 0}:
        mu = min(u, 2 * 10**6)
        engine.table_build(u, dense, mu)
        got = engine.table_checksums()
        engine.table_build(u, dense, mu, dr_b200.Params(segment_log2=18, block_threads=1024))
        assert got == engine.table_checksums(), (u, dense)


def test_default_shape_streamed(engine):
    X = 10**12
    p = dr_b200.default_params(X, dr_b200.POLICY_COMPRESSED)
    assert p.u_total < 150000000 and p.segment_log2 == 0
    try:
        whole = engine.mertens(X, p)
        for resident, band in ((2 * 10**7, 3 * 10**6), (1.2e7, 0)):
            engine.set_resident_limit(int(resident), band)
            r = engine.mertens(X, p)
            assert r.stats.bands > 0
            assert (r.M, r.stats.C, r.stats.S1, r.stats.S2) == (62366, whole.stats.C, whole.stats.S1, whole.stats.S2)
    finally:
        engine.set_resident_limit(0)
