"""GPU: dr_table_build_noalloc's odd mode (segments above 2 u_dense, any u_dense).

Odd and even dense cutoffs on and off 64-value words, none at all, cutoffs near half the table
(hardly an odd segment), a last segment of a few values and table sizes around the switch to
large segments: every buffer bit for bit as dr_table_build makes it (its checksums, and M(n)
read back from it)."""
import ctypes

import numpy as np
import pytest

import dr_b200

pytestmark = pytest.mark.gpu

CASES = [(149999999, 1000), (150000000, 1001), (200000003, 0), (200000003, 64), (260000001, 12345677),
         (260000002, 12345678), (300000007, 140000001), (300000007, 149999999), (400000000 + (1 << 18) + 3, 1 << 18),
         (1000000033, 4000003), (10**7 + 1, 33333)]


@pytest.mark.parametrize("ut,ud", CASES)
def test_odd_mode_tables(engine, ut, ud):
    import torch

    ml = min(ut, 3 * 10**6)
    W = (ut - ud + 63) // 64
    G = ml // 192 + 2
    dM = torch.empty(max(ud, 8), dtype=torch.int16, device="cuda")
    planes = torch.full((2 * W,), -1, dtype=torch.int64, device="cuda")
    ckpt = torch.full((W,), -1, dtype=torch.int32, device="cuda")
    wheel = torch.full((4 * G,), -1, dtype=torch.int32, device="cuda")
    p = ctypes.c_void_p
    rc = dr_b200.lib().dr_table_build_noalloc(0, p(torch.cuda.current_stream().cuda_stream), ut, ud, ml,
                                              p(dM.data_ptr()), p(planes.data_ptr()), p(ckpt.data_ptr()),
                                              p(wheel.data_ptr()))
    assert rc == 0, dr_b200.lib().dr_last_error().decode()
    torch.cuda.synchronize()
    engine.table_build(ut, ud, ml)
    want = engine.table_checksums()
    k = torch.arange(W, dtype=torch.int64, device="cuda") * 2 + 1
    n = torch.arange(1, ud + 1, dtype=torch.int64, device="cuda") * 2 + 1
    d = dM[:ud].to(torch.int64)
    got = [int(d.sum()), int((d * n).sum()), int((planes[0::2] * k).sum()), int((planes[1::2] * k).sum()),
           int((ckpt.to(torch.int64) * k).sum())]
    assert [v % 2**64 for v in got] == [want[0], want[1], want[3], want[4], want[5]]
    # the wheel: mu of j = 6m + 1 and 6m + 5
    m = np.arange(0, (ml - 5) // 6)
    w = wheel.cpu().numpy().view(np.uint32).reshape(-1, 4)
    mu = engine.table_read_wheel(0, ml + 1)
    for c, j in ((0, 6 * m + 1), (2, 6 * m + 5)):
        nz, ng = (w[m >> 5, c] >> (m & 31)) & 1, (w[m >> 5, c + 1] >> (m & 31)) & 1
        assert np.array_equal(nz.astype(np.int8) * (1 - 2 * ng.astype(np.int8)), mu[j])
