"""The far field's CTAs as the kernel decodes them, on the host (no GPU):
gi_debug_pair_task runs the kernel's own decode of one CTA of a run.  Every
unordered pair must be some warp's exactly once, and no warp of the far field's
finer split may be without pairs."""
from __future__ import annotations

import numpy as np
import pytest

CHUNK = 64


def _cover(gi, n, pcl, potential):
    """How often each pair i < j is evaluated: a warp has rows r0 .. r0 + rows and the
    chunks [c0, c1); it keeps i < j, and no chunk that ends before its rows."""
    count = np.zeros((n, n), np.uint8)
    tasks, empty = gi.pair_tasks(n, pcl, potential), 0
    for r0, rows, c0, c1 in tasks:
        assert r0 % rows == 0
        empty += c0 >= c1
        i, j = np.arange(r0, min(r0 + rows, n)), np.arange(c0 * CHUNK, min(c1 * CHUNK, n))
        if len(i) and len(j):
            assert c0 * CHUNK >= r0  # the kernel's diagonal rule covers the rest
            count[np.ix_(i, j)] += (i[:, None] < j[None, :]).astype(np.uint8)
    return count, tasks, empty


@pytest.mark.parametrize("potential", [False, True])
@pytest.mark.parametrize("pcl", [-1, 0, 2, 4])
@pytest.mark.parametrize("n", [1, 64, 65, 129, 1000, 1025, 2049, 3072, 3073, 4000, 6145])
def test_every_pair_once(gi, n, pcl, potential):
    count, tasks, empty = _cover(gi, n, pcl, potential)
    upper = np.triu(np.ones((n, n), bool), 1)
    assert (count[upper] == 1).all() and (count[~upper] == 0).all()
    if pcl < 0 and not potential:
        assert empty == 0


@pytest.mark.parametrize("n", [12287, 12288, 20011, 32767, 32768, 65535, 65536, 131072])
@pytest.mark.parametrize("potential", [False, True])
def test_default_split_by_chunks(gi, n, potential):
    """The same at sizes where pairs are too many to list: each group of 64 rows takes
    every chunk from its own on once."""
    chunks = -(-n // CHUNK)
    count = np.zeros((chunks, chunks), np.uint8)
    for r0, rows, c0, c1 in gi.pair_tasks(n, -1, potential):
        g = np.arange(r0 // CHUNK, min((r0 + rows) // CHUNK, chunks))
        if c0 < c1 and len(g):
            count[g[0]:g[-1] + 1, c0:c1] += 1
    upper = np.triu(np.ones((chunks, chunks), bool))
    assert (count[upper] == 1).all()


@pytest.mark.parametrize("n", [8448000, 24000000, 100000000, 2000000000])
def test_potential_of_many_bodies(gi, n):
    """The potential's tasks are numbered in 64 bits (its CTAs take several each): the
    first and last of them have pairs of the run."""
    total = gi.pair_task_count(n, -1, True)
    chunks = -(-n // CHUNK)
    assert total * 256 * 512 >= n * (n - 1) // 2  # rows and bodies of 8 chunks a task
    for k in (0, 1, 3, total // 2, total - 1):
        r0, rows, c0, c1 = gi.pair_task(n, -1, True, k)
        assert rows == 256 and 0 <= r0 < n + 1024 and r0 // CHUNK <= max(c0, r0 // CHUNK) and c1 <= chunks
