"""gi_potential_fp64 above 12,288 bodies: states so wide that a place past the run's
end would count."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n", [12545, 12608, 12799])
def test_no_pairs_past_the_run(gi, orc, torch_cuda, n):
    """Bodies 1e14 apart (pairs of 1e-14), the run ending inside a group of 256:
    the staged places past its end, at 1e16, count for nothing."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    pos, _, _ = gi.ic_uniform_ball(n, n, 1.0)
    pos[:, :3] *= np.float32(1e14)
    run = wl.run_desc(gi, 0, n, 900)
    ctx = gi.Context(0)
    got = ctx.potential(_dev(torch, pos).data_ptr(), [run], p)[0]
    ctx.close()
    want = orc.potential_fp64(pos, [run], p).sum() / 2.0
    assert abs(got - want) <= 2e-7 * abs(want)
