"""GPU: dr_stats.kernel_launches is the number of kernels that ran (memory sets and copies apart),
as the profiler counts them: every route of a call, eager and replayed."""
import pytest

import dr_b200

pytestmark = pytest.mark.gpu


def _kernels(call):
    """The kernels of one call by the profiler's count, and the call's result."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        r = call()
        torch.cuda.synchronize()
    return sum(1 for e in prof.events() if "_kernel" in e.name or "scan_" in e.name), r


def _counts(call, stats):
    call()  # buffers, modules
    n, r = _kernels(call)
    assert n > 0
    return n, stats(r).kernel_launches


CALLS = {
    "from the table": (10**6, dr_b200.default_params(10**6), None),  # one segment launch, direct
    "one-CTA scan": (10**9, dr_b200.default_params(10**9), None),
    "three-pass scan": (10**14, dr_b200.default_params(10**14, dr_b200.POLICY_DENSE), None),
    "buckets, odd mode, windows": (10**15, dr_b200.default_params(10**15, dr_b200.POLICY_COMPRESSED), None),
    "windowed S1": (10**13, dr_b200.Params(**{**dr_b200.default_params(10**13, dr_b200.POLICY_GPU).as_dict(),
                                              "s1_window_log2": 12}), None),
    "above 2^51": ((1 << 51) + 12345, dr_b200.Params(u_total=400000000, u_dense=100000000, cx=1.25,
                                                     mu_limit=100000000), None),
    "streamed": (10**13, dr_b200.default_params(10**13, dr_b200.POLICY_COMPRESSED), (42000000, 10**7)),
}


@pytest.mark.parametrize("name", list(CALLS))
def test_single_query(name):
    X, p, resident = CALLS[name]
    with dr_b200.Engine(0) as e:
        if resident:
            e.set_resident_limit(*resident)
        n, counted = _counts(lambda: e.mertens(X, p), lambda r: r.stats)
    assert n == counted


def test_table_build(engine):
    for u, d in ((10**6, 10**6), (2 * 10**9, 10**8)):
        n, counted = _counts(lambda: engine.table_build(u, d, 10**6), lambda st: st)
        assert n == counted, u


def test_replayed_batch():
    xs = [10**9 + k for k in range(20)] + [10**11, 10**6]
    with dr_b200.Engine(0) as e:
        eager = e.mertens_batch(xs)[1].kernel_launches
        n, counted = _counts(lambda: e.mertens_batch(xs), lambda r: r[1])
    assert n == counted == eager
