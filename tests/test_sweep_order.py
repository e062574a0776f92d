"""The order in which a batch's full sweep claims its work items (sweep_item in
gdp_batch.cu), restated on the CPU: every item of every unit exactly once, each
unit's items in their order, and an equal part of every unit's list at a time."""
import numpy as np
import pytest

PARTS = 8


def sweep_item(prefix, i):
    total = prefix[-1]
    q, rem = divmod(total, PARTS)
    s = i // (q + 1) if i < rem * (q + 1) else rem + (i - rem * (q + 1)) // q
    i -= s * q + min(s, rem)
    below = lambda x: (x + PARTS - 1 - s) // PARTS
    before = lambda x: x // PARTS * s + min(s, x % PARTS)
    lo, hi = 0, len(prefix) - 2
    while lo < hi:
        mid = (lo + hi + 1) >> 1
        if below(prefix[mid]) <= i:
            lo = mid
        else:
            hi = mid - 1
    return lo, before(prefix[lo + 1]) - before(prefix[lo]) + i - below(prefix[lo])


@pytest.mark.parametrize("sizes", [[1], [7], [8], [9], [1, 1, 1], [3, 0, 5], [0, 0, 1], [17, 4, 100, 1, 33],
                                   [1000, 2, 2, 2], list(range(40))])
def test_every_item_once(sizes):
    prefix = [0] + [int(x) for x in np.cumsum(sizes)]
    got = [sweep_item(prefix, i) for i in range(prefix[-1])]
    assert sorted(got) == [(k, a) for k, n in enumerate(sizes) for a in range(n)]
    for k in range(len(sizes)):
        mine = [a for u, a in got if u == k]
        assert mine == sorted(mine)
    # after c of the claims each unit is at its share of them, up to a part and a few items
    done = [0] * len(sizes)
    for c, (k, a) in enumerate(got, 1):
        done[k] = a + 1
        assert all(abs(d - n * c / prefix[-1]) <= n / PARTS + 3 for d, n in zip(done, sizes))
