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
