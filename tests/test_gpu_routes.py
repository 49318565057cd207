"""GPU: the kernel that takes the sums of a launch, on both sides of the rule.

Launches of little work, and queries of few candidates on a large table, go to the sums kernel,
the rest to tiles; the sums are the same either way (a query alone with the windowed S1 asked for
never takes tiles)."""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu


def _kernels(call):
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        r = call()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    return {k for k in ("tiles_kernel", "sums_kernel") if any(k in n for n in names)}, r


@pytest.mark.parametrize("count,u,N,takes", [
    (1, 10**5, 5, "tiles_kernel"), (1, 10**5, 1000, "tiles_kernel"), (1, 5 * 10**8, 1000, "sums_kernel"),
    (1, 2 * 10**7, 20000, "tiles_kernel"), (300, 2 * 10**7, 30, "sums_kernel"), (300, 2 * 10**7, 600, "tiles_kernel"),
    (300, 5 * 10**8, 30, "sums_kernel"), (300, 5 * 10**8, 1000, "tiles_kernel"), (40, 10**6, 4, "tiles_kernel")])
def test_route(engine, count, u, N, takes):
    X, cx = u * N + u // 2, 1.25
    xs = [X + 7 * k for k in range(count)]
    mu = max(int(cx * xs[-1] ** 0.5) + 2, N + 2)
    p = dr_b200.Params(u_total=max(u, mu), u_dense=max(u // 4, mu), cx=cx, mu_limit=mu)
    ps = [p] * count
    engine.mertens_batch(xs, ps)
    used, (out, _) = _kernels(lambda: engine.mertens_batch(xs, ps))
    assert used == {takes}
    sums = engine.batch_checksums(count)
    q = dr_b200.Params(**{**p.as_dict(), "s1_window_log2": 12})
    for k in sorted({0, count // 2, count - 1}):
        used, r = _kernels(lambda: engine.mertens(xs[k], q))
        assert p.u_dense < 2 * 4096 or used == {"sums_kernel"}
        assert (out[k],) + tuple(sums[k]) == (r.M, r.stats.C, r.stats.S1, r.stats.S2)
