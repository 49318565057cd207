"""GPU: a resident limit bounds what a streamed call holds.

The plane words that bands keep for the ones above may take at most half of what the resident
table and the band buffers take; they go back to the device when the limit changes."""
import gc

import pytest

import dr_b200

pytestmark = pytest.mark.gpu


def _used():
    import torch

    gc.collect()  # no context of an earlier test
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def _limit_bytes(u_dense, resident, band):
    return 2 * u_dense + 20 * (resident - u_dense + band) // 64


def _call(resident, band, u_dense):
    X = 10**15
    p = dr_b200.default_params(X, dr_b200.POLICY_GPU)
    p.u_dense = u_dense
    with dr_b200.Engine(0) as e:
        e.mertens(10**9)  # modules and the launch of each kernel
        base = _used()
        e.set_resident_limit(resident, band)
        r = e.mertens(X, p)
        held = _used() - base
        e.set_resident_limit(0)
        return r, held, held - (_used() - base)


def test_small_limit_keeps_no_words():
    """6e7 of 4.9e9 values resident: the words of 2.4e9 values (0.6 GB) would be four times
    the limit's own 0.15 GB.  What the call needs besides the table is under 0.7 GB."""
    dense, resident, band = 40000000, 60000000, 2 * 10**8
    r, held, back = _call(resident, band, dense)
    assert r.M == -3216373 and r.stats.bands > 20
    assert held < 1.5 * _limit_bytes(dense, resident, band) + 0.7e9
    assert back == 0


def test_kept_words_go_back_with_the_limit():
    dense, resident, band = 4 * 10**8, 2 * 10**9, 10**9
    r, held, back = _call(resident, band, dense)
    assert r.M == -3216373 and r.stats.bands == 3
    kept = 16 * 10**9 // 64  # one band below u/2
    assert 2 * kept <= _limit_bytes(dense, resident, band)
    assert abs(back - kept) < 8 << 20
