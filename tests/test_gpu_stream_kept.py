"""GPU: bands of a streamed table in odd mode from the plane words that earlier bands keep.

Bands above twice the resident table find the halves of their even values in the kept words
of the bands below u_total/2.  Same sums as the whole table for bands of many lengths (halves
in the resident table, across its end, in one kept band, across two), and under memory budgets
that leave room for the kept words or not."""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu


def _sums(r):
    return r.M, r.stats.C, r.stats.S1, r.stats.S2


@pytest.mark.parametrize("lg", [14, 18])
def test_kept_bands(engine, lg):
    X = 10**13
    p = dr_b200.default_params(X, dr_b200.POLICY_COMPRESSED)
    p.segment_log2 = lg
    p.u_dense = 20000000 // 64 * 64
    try:
        whole = _sums(engine.mertens(X, p))
        assert whole[0] == 599582
        for resident, band in ((42000000, 3000001), (45000000, 10**7), (41000000, 2 * 10**7 + 5), (60000000, 0),
                               (10**8, 1), (21000000, 5 * 10**6)):
            if band == 1 and lg == 14:
                band = 1 << 17
            engine.set_resident_limit(resident, band)
            r = engine.mertens(X, p)
            assert r.stats.bands > 1 and _sums(r) == whole, (resident, band)
    finally:
        engine.set_resident_limit(0)


def test_budgets():
    X = 10**15
    p = dr_b200.default_params(X, dr_b200.POLICY_GPU)
    with dr_b200.Engine(0) as e:
        want = _sums(e.mertens(X, p))
    done = 0
    for mb in range(1000, 2600, 100):
        with dr_b200.Engine(0) as e:
            e.set_hbm_budget(mb << 20)
            e.set_resident_limit(10**9, 4 * 10**8)
            try:
                assert _sums(e.mertens(X, p)) == want
                done += 1
            except dr_b200.DRError as err:
                assert err.code == dr_b200.DR_ERR_NOMEM
    assert done > 2
