"""Batches of short runs, whose contacts go through a cell grid that the run alone
does without: the same bits either way, with the grids built by clusters and by the
grid-wide kernels, beside the far field and on one stream."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_contact_paths import _aliased, _dev

pytestmark = pytest.mark.gpu


def _batch(sizes, seed):
    """Runs of the given sizes, sparse, settled, crowded and aliased in turn."""
    rng = np.random.default_rng(seed)
    parts = []
    for k, n in enumerate(sizes):
        if k % 4 == 3 and n > 16:
            parts.append(_aliased(seed + k, n))
            continue
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        rho = (0.25, 4.0, 540.0)[k % 4 % 3]
        pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
        pos[:, :3] = d * (3 * n / (4 * np.pi * rho)) ** (1 / 3) * rng.uniform(size=(n, 1)) ** (1 / 3)
        vel[:, :3] = rng.normal(scale=1.5, size=(n, 3))
        parts.append((pos, vel))
    return [np.concatenate([p[k] for p in parts]) for k in (0, 1)]


@pytest.mark.parametrize("accum", ["PAIRED", "KAHAN"])
@pytest.mark.parametrize("sizes", [[3500, 513, 600, 3499], [1, 512, 513, 31, 1000, 1023, 1024, 1025] * 3 + [3000, 3400],
                                   [2047, 2048, 2049, 2050] * 6, [900, 1800] * 32, [3501, 700, 4096, 4097, 2000],
                                   [30000, 2000, 2500, 3000, 1500]])
def test_batch_equals_runs_alone(gi, orc, torch_cuda, sizes, accum):
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    assert any(gi.contact_plan(sizes))
    pos, vel = _batch(sizes, len(sizes))
    off = np.concatenate([[0], np.cumsum(sizes)])
    runs = [wl.run_desc(gi, int(o), n, n // 5) for o, n in zip(off, sizes)]
    dp, dv = _dev(torch, pos), _dev(torch, vel)
    ctx = gi.Context(0, accum=getattr(gi, "GI_ACCUM_" + accum))
    both, alone = torch.zeros_like(dp), torch.zeros_like(dp)
    ctx.forces(dp.data_ptr(), dv.data_ptr(), both.data_ptr(), runs, p)
    for r in runs:
        ctx.forces(dp.data_ptr(), dv.data_ptr(), alone.data_ptr(), [r], p)
    torch.cuda.synchronize()
    ctx.close()
    assert torch.equal(both, alone)
    got = both.cpu().numpy()
    for r in runs[:5]:
        if r.n > 1:
            one = wl.run_desc(gi, 0, r.n, r.nfe)
            s = slice(r.offset, r.offset + r.n)
            idx = np.unique(np.linspace(0, r.n - 1, 64).astype(np.int32))
            f64, _ = orc.forces_fp64(pos[s], vel[s], [one], p, idx=idx)
            assert rel_l2(got[s][idx, :3], f64) < 1e-5
