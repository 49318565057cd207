"""GPU: dr_table_build_noalloc of a few segments, on both sides of the change of shape: every
buffer as dr_table_build makes it (its checksums and mu of the wheel)."""
import ctypes

import numpy as np
import pytest

import dr_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ut", [1, 63, 1000, 32768, 32769, 65535, 65536, 65537, 65600, 131073])
def test_small_tables(engine, ut):
    import torch

    p = ctypes.c_void_p
    for ud in sorted({0, ut // 3, ut // 3 // 64 * 64, ut}):
        ml = ut
        W, G = (ut - ud + 63) // 64, ml // 192 + 2
        dM = torch.empty(max(ud, 8), dtype=torch.int16, device="cuda")
        planes = torch.full((max(2 * W, 2),), -1, dtype=torch.int64, device="cuda")
        ckpt = torch.full((max(W, 1),), -1, dtype=torch.int32, device="cuda")
        wheel = torch.full((4 * G,), -1, dtype=torch.int32, device="cuda")
        rc = dr_b200.lib().dr_table_build_noalloc(0, p(torch.cuda.current_stream().cuda_stream), ut, ud, ml,
                                                  p(dM.data_ptr()), p(planes.data_ptr()), p(ckpt.data_ptr()),
                                                  p(wheel.data_ptr()))
        assert rc == 0, dr_b200.lib().dr_last_error().decode()
        torch.cuda.synchronize()
        engine.table_build(ut, ud, ml)
        want = engine.table_checksums()
        k = torch.arange(W, dtype=torch.int64, device="cuda") * 2 + 1
        n = torch.arange(1, ud + 1, dtype=torch.int64, device="cuda") * 2 + 1
        d, pl, ck = dM[:ud].to(torch.int64), planes[: 2 * W], ckpt[:W].to(torch.int64)
        got = [int(d.sum()), int((d * n).sum()), int((pl[0::2] * k).sum()), int((pl[1::2] * k).sum()),
               int((ck * k).sum())]
        assert [v % 2**64 for v in got] == [want[0], want[1], want[3], want[4], want[5]], ud
        m = np.arange(0, max(0, (ml - 5) // 6 + 1))
        w = wheel.cpu().numpy().view(np.uint32).reshape(-1, 4)
        mu = engine.table_read_wheel(0, ml + 1)
        for c, j in ((0, 6 * m + 1), (2, 6 * m + 5)):
            nz, ng = (w[m >> 5, c] >> (m & 31)) & 1, (w[m >> 5, c + 1] >> (m & 31)) & 1
            assert np.array_equal(nz.astype(np.int8) * (1 - 2 * ng.astype(np.int8)), mu[j]), ud
