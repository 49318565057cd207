"""GPU: the window kernel (csrc/dr_windows.cu).

It takes the near S1 lookups of large launches from windows of 98304 table values; the rest
stays with the tile kernel.  How many windows there are follows from the dense tier, so C, S1
and S2 must not change with it: none, less than one window, one, several and all of them.
Also a batch whose queries share the windows, split points and table sizes away from the
defaults, and a memory budget so tight that the window kernel's own buffers do not fit.
"""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu
W = 98304


def _sums(r):
    return r.M, r.stats.C, r.stats.S1, r.stats.S2, r.stats.s1_ops, r.stats.s2_ops


def test_dense_tier_sizes(engine):
    X = 10**15
    p = dr_b200.default_params(X, dr_b200.POLICY_COMPRESSED)
    want = _sums(engine.mertens(X, p))
    assert want[0] == -3216373
    for dense in (0, W - 1, W, W + 64, 3 * W + 8, 20 * W - 1, p.u_total // 2 // 64 * 64 + 7):
        q = dr_b200.Params(**{**p.as_dict(), "u_dense": dense})
        assert _sums(engine.mertens(X, q)) == want, dense


@pytest.mark.parametrize("cx,fu", [(0.4, 1.0), (0.9, 0.3), (2.5, 2.0), (6.0, 0.6)])
def test_splits_match_single_evaluations(engine, cx, fu):
    X = 2 * 10**15 + 12345
    p = dr_b200.default_params(X, dr_b200.POLICY_GPU)
    mu = int(cx * X**0.5) + 2000
    u = max(int(p.u_total * fu), mu + 64)
    mu = min(u, max(mu, X // u + 1000))
    q = dr_b200.Params(u_total=u, u_dense=min(u, p.u_dense), cx=cx, mu_limit=mu)
    got = _sums(engine.mertens(X, q))
    q.s1_window_log2 = 12  # every lookup and position in the windowed S1 and the sums kernel
    assert got == _sums(engine.mertens(X, q))


def test_batch_shares_windows(engine):
    xs = [10**15 + 7, 3 * 10**12, 10**9, 5 * 10**14 + 1, 10**15 + 7, 8 * 10**13]
    p = dr_b200.default_params(max(xs), dr_b200.POLICY_COMPRESSED)
    out, _ = engine.mertens_batch(xs, [p] * len(xs))
    again, _ = engine.mertens_batch(xs, [p] * len(xs))  # replayed from its graph
    sums = engine.batch_checksums(len(xs))
    assert out == again
    for x, m, c in zip(xs, out, sums):
        assert (m,) + tuple(c) == _sums(engine.mertens(x, p))[:4], x


def test_tight_budget():
    X = 10**15
    p = dr_b200.default_params(X, dr_b200.POLICY_COMPRESSED)
    need = dr_b200.query_bytes(X, p)
    lo, hi = int(need * 0.9), int(need * 1.1)  # the smallest budget that works lies between
    while hi - lo > 65536:
        mid = (lo + hi) // 2
        with dr_b200.Engine(0) as e:
            e.set_hbm_budget(mid)
            try:
                assert e.mertens(X, p).M == -3216373
                hi = mid
            except dr_b200.DRError as err:
                assert err.code == dr_b200.DR_ERR_NOMEM
                lo = mid
    assert hi < int(need * 1.1)
