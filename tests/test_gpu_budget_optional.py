"""GPU: memory budgets between what a call needs and what its fastest form would like.

The smallest budget that a fresh context accepts must be the one of the buffers that the call
cannot do without: what only speeds it up is reserved last and given up there."""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu

M_1E15 = -3216373  # test_dr.cpp:26-47


def _run(X, p, budget, resident=None):
    """The result on a fresh context under the budget; None where it does not fit."""
    with dr_b200.Engine(0) as e:
        if budget:
            e.set_hbm_budget(budget)
        if resident:
            e.set_resident_limit(*resident)
        try:
            return e.mertens(X, p)
        except dr_b200.DRError as err:
            assert err.code == dr_b200.DR_ERR_NOMEM
            return None


def _smallest(X, p, lo, hi):
    while hi - lo > 256:
        mid = (lo + hi) // 2
        if _run(X, p, mid):
            hi = mid
        else:
            lo = mid
    return hi


def test_window_buffers_are_given_up():
    """At the smallest budget the window kernel's buffers do not fit: one launch fewer."""
    X = 10**15
    p = dr_b200.default_params(X, dr_b200.POLICY_COMPRESSED)
    need = dr_b200.query_bytes(X, p)
    tight, ample = _run(X, p, _smallest(X, p, need // 2, need * 2)), _run(X, p, 0)
    assert tight.M == ample.M == M_1E15
    assert tight.stats.kernel_launches == ample.stats.kernel_launches - 1
    for f in ("C", "S1", "S2", "s1_ops", "s2_ops"):
        assert getattr(tight.stats, f) == getattr(ample.stats, f)


# Budgets (bytes) that held these calls when every evaluation had its own record and no tile
# kernel existed: the per-slot calls (X >= 2^51, a streamed table) and queries of one or two
# candidates each, whose tile records would come on top.
REST = dr_b200.Params(u_total=400000000, u_dense=100000000, cx=1.25, mu_limit=100000000)


@pytest.mark.parametrize("X,p,resident,budget", [
    ((1 << 51) + 12345, REST, None, 1444223596),
    (3 * 10**15, dr_b200.default_params(3 * 10**15, dr_b200.POLICY_GPU), None, 5155890772),
    (10**13, dr_b200.default_params(10**13, dr_b200.POLICY_COMPRESSED), (42000000, 10**7), 158101253),
    (10**15, dr_b200.default_params(10**15, dr_b200.POLICY_GPU), (10**9, 4 * 10**8), 1448320307),
])
def test_tile_records_are_given_up(X, p, resident, budget):
    ample = _run(X, p, 0, resident)
    assert dr_b200.query_bytes(X, p) >= budget  # what the checks promise is enough
    for b in (budget, dr_b200.query_bytes(X, p)):
        r = _run(X, p, b, resident)
        assert r is not None, b
        for f in ("M", "C", "S1", "S2", "s1_ops", "s2_ops", "terms", "evals", "s1_comp_ops"):
            assert getattr(r.stats, f) == getattr(ample.stats, f), (b, f)


def test_batch_of_short_queries():
    import random

    rng = random.Random(1)
    xs = [10**6 + rng.randrange(1, 3 * 10**6) for _ in range(20000)]
    ps = [dr_b200.Params(u_total=10**6, u_dense=10**6, cx=1.0, mu_limit=10000)] * len(xs)
    with dr_b200.Engine(0) as e:
        want = e.mertens_batch(xs, ps)[0]
    with dr_b200.Engine(0) as e:
        e.set_hbm_budget(9332800)
        for _ in range(3):  # eager, then replayed
            assert e.mertens_batch(xs, ps)[0] == want
