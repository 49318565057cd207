"""GPU: the tile kernel's S1/S2 sums at the edges of its range.

The sums kernel, one evaluation at a time, is the second route: with the windowed S1 on it
takes every lookup the windows leave and every S2 position.  Same M, C, S1, S2 and counts
either way -- below, at and above X = 2^51 (from there on the smallest k go to the sums
kernel), with tables that put every lookup in the compressed tier, and at split points far
from the default, where some evaluations fall outside the tile kernel's domain (checked
against the oracle there).
"""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu

FIELDS = ("C", "S1", "S2", "s1_ops", "s2_ops", "terms", "evals", "s1_comp_ops")


def _all(r):
    return (r.M,) + tuple(getattr(r.stats, f) for f in FIELDS)


@pytest.mark.parametrize("X", [10**8 + 9, 10**11 + 1, (1 << 51) - 1, 1 << 51, (1 << 51) + 12345, 5 * (1 << 51) + 7])
def test_tiles_match_single_evaluations(engine, X):
    p = dr_b200.default_params(X, dr_b200.POLICY_GPU)
    p.s1_window_log2 = 12
    want = _all(engine.mertens(X, p))
    p.s1_window_log2 = 0
    assert _all(engine.mertens(X, p)) == want


@pytest.mark.parametrize("cx,u,dense", [(0.03, 60000, 60000), (0.3, 40000, 1), (1.0, 31700, 0), (5.0, 200000, 777),
                                        (17.0, 600000, 300000), (40.0, 1300000, 64)])
def test_split_points_vs_oracle(engine, oracle, cx, u, dense):
    for X in (10**8 + 7, 10**9 + 123):
        mu = max(int(cx * X**0.5) + 2, X // u + 2)
        if mu > u:
            u = mu
        q = dr_b200.Params(u_total=u, u_dense=dense, cx=cx, mu_limit=mu)
        assert dr_b200.check_params(X, q) == 0
        r, o = engine.mertens(X, q), oracle.run(X, u, dense, cx, mu)
        assert (r.M, r.stats.C, r.stats.S1, r.stats.S2) == (o["M"], o["C"], o["S1"], o["S2"])


def test_uneven_batch_matches_single_queries(engine):
    """Queries from a few candidates to many blocks of them, groups of every size, one launch."""
    xs = [10**7 + 1, 10**9, 3 * 10**9, 10**10 + 3, 10**11, 2 * 10**12 + 1]
    p = dr_b200.default_params(10**12, dr_b200.POLICY_COMPRESSED)
    ps = [dr_b200.Params(u_total=200000 + 1000 * i, u_dense=5000, cx=0.5 + 0.1 * i, mu_limit=p.u_total // 4)
          for i in range(len(xs))]
    for q, x in zip(ps, xs):
        q.u_total = max(q.u_total, int(q.cx * x**0.5) + 1000)
        q.mu_limit = min(q.u_total, max(int(q.cx * x**0.5) + 2, x // q.u_total + 2))
    top = max(max(q.mu_limit, x // q.u_total + 2) for q, x in zip(ps, xs))
    for q in ps:
        q.u_total = max(q.u_total, top)
        q.mu_limit = top
    out, _ = engine.mertens_batch(xs, ps)
    sums = engine.batch_checksums(len(xs))
    for x, q, m, c in zip(xs, ps, out, sums):
        r = engine.mertens(x, q)
        assert (m,) + tuple(c) == (r.M, r.stats.C, r.stats.S1, r.stats.S2), x
