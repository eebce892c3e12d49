"""Captured steps on the paths that launch their kernels early: one stream with a cell
grid, and a table of short runs after one whose contacts ran beside its far field."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_short_runs import _batch
from test_gpu_contact_paths import _dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[3649], [4097], [5477], [3400, 3400], [700] * 20, [1500, 5000],
                                   [2000] * 64 + [300] * 6, [300] * 64 + [9000] * 3])
def test_graph_matches_eager_steps(gi, torch_cuda, sizes):
    """Eight steps by two launches of a four-step graph, an eager call between them,
    against eight eager steps and the first and last run's steps alone."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    pos, vel = _batch(sizes, 7)
    off = np.concatenate([[0], np.cumsum(sizes)])
    runs = [wl.run_desc(gi, int(o), n, n // 5) for o, n in zip(off, sizes)]
    ends = runs[:1] + runs[1:][-1:]
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        s = st.cuda_stream
        eager = [_dev(torch, pos), _dev(torch, vel), torch.zeros(len(pos), 4, device="cuda"),
                 torch.zeros(len(pos), 4, device="cuda")]
        graphed, single = [t.clone() for t in eager], [t.clone() for t in eager]
        force = torch.zeros_like(eager[0])
        ctx = gi.Context(0)
        q = [t.data_ptr() for t in eager]
        ctx.step_pingpong(*q, runs, p, 8, s)
        g = ctx.graph(*[t.data_ptr() for t in graphed], runs, p, 4, s)
        g.launch(s)
        ctx.forces(graphed[0].data_ptr(), graphed[1].data_ptr(), force.data_ptr(), runs[:1], p, s)
        g.launch(s)
        q = [t.data_ptr() for t in single]
        for r in ends:
            ctx.step_pingpong(*q, [r], p, 8, s)
        st.synchronize()
        g.close()
        ctx.close()
    assert torch.equal(eager[0], graphed[0]) and torch.equal(eager[1], graphed[1])
    for r in ends:
        k = slice(r.offset, r.offset + r.n)
        assert torch.equal(eager[0][k], single[0][k]) and torch.equal(eager[1][k], single[1][k])
