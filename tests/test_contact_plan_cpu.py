"""Which runs of a call the contact pass builds a grid for (host arithmetic, no GPU):
testing every pair of a short run is the cheaper way only while all of them
together have few."""
from __future__ import annotations

import pytest

DIRECT, CANDIDATES = 4096, 3648 ** 2


@pytest.mark.parametrize("sizes", [[1], [3648], [3649], [4096], [2000, 2000, 2000], [2000, 2000, 2000, 2000],
                                   [500] * 48, [500] * 64, [1000] * 13, [1000] * 14, [4000] * 64,
                                   [66000] + [4000] * 63, [66000, 3000], [512] * 63 + [513], [1, 600, 3000, 20000]])
def test_candidates_are_bounded(gi, sizes):
    plan = gi.contact_plan(sizes)
    tested = sum(n * n for n, b in zip(sizes, plan) if b == 0)
    # at most one run of 3,648 bodies, or 64 of 512 where there are more short runs
    assert tested <= max(CANDIDATES, 64 * 512 ** 2)
    short = sum(n * n for n in sizes if n <= DIRECT)
    for n, b in zip(sizes, plan):
        assert (b == 0) == (n <= (DIRECT if short <= CANDIDATES else 512))
        if b:  # a power of two in (n, 2 n], at least 8 cells a side
            assert n < b <= 2 * n and b & (b - 1) == 0 and b >= 1024
