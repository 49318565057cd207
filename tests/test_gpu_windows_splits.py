"""GPU: the window kernel at split parameters far from the defaults.

Divisor ranges there are much longer or shorter than at cx near 1; the second route is the
windowed S1 with the sums kernel, which takes every lookup and position.  A call whose planned
window lookups are not all summed is an error, so that these pass says that none was lost."""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu

FIELDS = ("C", "S1", "S2", "s1_ops", "s2_ops", "terms", "evals", "s1_comp_ops")


def _sums(r):
    return (r.M,) + tuple(getattr(r.stats, f) for f in FIELDS)


@pytest.mark.parametrize("X,cx,u,dense", [
    (10**13 + 7, 0.01, 10**9, 5 * 10**8), (10**13 + 7, 0.03, 10**9, 10**9), (2 * 10**13 + 1, 0.0624, 2 * 10**9, 10**8),
    (10**14 + 3, 0.0626, 2 * 10**9, 10**9),
    (10**14 + 3, 0.31, 10**9, 10**9), (2 * 10**15 + 9, 16.5, 7.5e8, 4 * 10**8), (2 * 10**15 + 5, 17.0, 8 * 10**8, 98304 * 7 + 3)])
def test_extreme_splits(engine, X, cx, u, dense):
    mu = max(int(cx * X**0.5) + 2, X // int(u) + 2)
    p = dr_b200.Params(u_total=int(u), u_dense=int(dense), cx=cx, mu_limit=mu)
    assert dr_b200.check_params(X, p) == 0
    got = engine.mertens(X, p)
    assert bool(dr_b200.window_items(X, p)) == (cx >= 0.3)  # work enough for the window kernel
    p.s1_window_log2 = 12
    assert _sums(got) == _sums(engine.mertens(X, p))
