"""CPU: the window kernel's items cover every lookup that the planner leaves to it.

The planner leaves out of the tile kernel the S1 lookups M(y // n) of a block of 32 candidates
whose quotient lies in the first tile_windows(block) windows of 98304 values; the host's items
name, per window, the blocks that the window kernel looks at.  They must be the blocks whose
windows include it, less leading ones whose smallest quotient lies above the window: that
quotient is worked out here from the split point as the planner does.  Split parameters over
the whole range that takes windows, far from the defaults above all.  Below 0.3 there are none:
long divisor ranges read the table as fast from the tile kernel, and one block of the first
candidates would hold a window's work for one CTA."""
import math
import random

import pytest

import dr_b200

W = 98304
WIN_RUN = 32.0  # odd divisors of the block's first candidate below which its windows stop


def _tile_windows(X, blk, twin_max):
    w = math.sqrt(float(X) / float(96 * blk + 1) * (1.0 / (2.0 * WIN_RUN * W)))
    return int(w) if w < float(twin_max) else twin_max


def _split(cx, y):
    return max(1, min(y - 1, int(cx * math.sqrt(float(y)))))


def _smallest_quotient(y, cx):
    """Over the S1 divisors of single(y) and comb2(y, y // 2)."""
    n = y // (_split(cx, y) + 1)
    y2 = y // 2
    if y2 > 1:
        n = max(n, 2 * (y2 // (_split(cx, y2) + 1)))
    return y // max(n, 1)


CASES = [(X, cx, u) for cx, sizes in (
    (0.3, ((10**14, 10**9), (10**16, 5 * 10**9))), (1.25, ((10**15, 5 * 10**9), (10**17, 10**11))),
    (6.0, ((10**15, 3 * 10**8), (10**17, 3 * 10**9))), (17.0, ((2 * 10**15, 8 * 10**8), (10**17, 6 * 10**9))),
    (40.0, ((10**16, 4 * 10**9), (10**17, 1.3 * 10**10))), (63.0, ((10**17, 2 * 10**10),))) for X, u in sizes]


@pytest.mark.parametrize("X,cx,u", CASES)
def test_items_cover_the_near_lookups(X, cx, u):
    rng = random.Random(int(X) + int(1000 * cx))
    X, u = X - rng.randrange(X // 1000), int(u)
    for dense in (min(u, 2 * 10**9), min(u, 5 * W + 7)):
        p = dr_b200.Params(u_total=u, u_dense=dense, cx=cx, mu_limit=u)
        items = dr_b200.window_items(X, p)
        # every case has window work, but where the first five windows lie below every quotient
        assert items or (dense < 10**6 and _smallest_quotient(u, cx) > 5 * W)
        # windows inside the dense tier and worth their staging (2^18 lookups in all)
        twin_max = int(min(math.sqrt(float(X) * W / (2.0 * 262144.0)), float(min(dense, 2**31 - 1))) / W)
        N = X // u
        nc = 2 * (N // 6) + (N % 6 >= 1) + (N % 6 >= 5)
        nb = (nc + 31) // 32
        by_w = {}
        for w, b0, b1 in items:
            by_w.setdefault(w, []).append((b0, b1))
        for w in range(_tile_windows(X, 0, twin_max)):
            hi = nb  # blocks whose windows include w: [0, hi)
            lo = 1
            while lo < hi:
                mid = (lo + hi + 1) // 2
                if _tile_windows(X, mid - 1, twin_max) > w:
                    lo = mid
                else:
                    hi = mid - 1
            runs = sorted(by_w.get(w, []))
            at = runs[0][0] if runs else hi
            assert runs == [] or (runs[-1][1] == hi and all(a[1] == b[0] for a, b in zip(runs, runs[1:]))), w
            if at == 0:
                continue
            last = 96 * at - 1  # the largest candidate of the skipped blocks
            for k in [last] + [rng.randrange(1, last + 1) for _ in range(20)]:
                for y in (X // k,) + ((X // k // 3,) if 3 * k <= N else ()):
                    assert _smallest_quotient(y, cx) >= (w + 1) * W, (w, k)


@pytest.mark.parametrize("X,cx,u", [(10**13, 0.01, 10**9), (10**13, 0.05, 10**9), (10**15, 0.1, 10**10),
                                    (10**14, 0.2, 10**9), (2 * 10**15, 0.2999, 10**10)])
def test_no_windows_for_long_ranges(X, cx, u):
    p = dr_b200.Params(u_total=u, u_dense=u // 8, cx=cx, mu_limit=u)
    assert dr_b200.window_items(X, p) == []
