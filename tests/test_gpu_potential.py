"""gi_potential_fp64 above 12,288 bodies: crowded states, whose contacts carry the
sum, and states so wide that a place past the run's end would count."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _coincident(wl, n, nfe):
    """The potential of n bodies in one point, and what the pair's own FP32
    arithmetic may leave: four roundings of at most 2^-24 of 2 G + 2 K / 3."""
    m = wl.MATERIAL
    nsi = n - nfe
    classes = [(nsi * (nsi - 1) // 2, m["mass_si"] ** 2, 2 * m["k_si"]),
               (nsi * nfe, m["mass_fe"] * m["mass_si"], m["k_fe"] + m["k_si"]),
               (nfe * (nfe - 1) // 2, m["mass_fe"] ** 2, 2 * m["k_fe"])]
    return (sum(c * (-2.0 * g + 2.0 * k / 3.0) for c, g, k in classes),
            sum(c * 4 * 2.0 ** -24 * (2.0 * g + 2.0 * k / 3.0) for c, g, k in classes))


@pytest.mark.parametrize("n,nfe", [(12289, 0), (12545, 12545), (13000, 4000)])
def test_coincident_bodies(gi, torch_cuda, n, nfe):
    """All bodies in one point: every pair of a class has the same potential, so
    that sums in FP32 would be off by the same rounding each time (2e-6 of a sum
    of 128 equal terms, 4e-6 of 512)."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = [0.25, -3.5, 7.0]
    ctx = gi.Context(0)
    got = ctx.potential(_dev(torch, pos).data_ptr(), [wl.run_desc(gi, 0, n, nfe)], p)[0]
    ctx.close()
    want, tol = _coincident(wl, n, nfe)
    assert abs(got - want) <= tol


@pytest.mark.parametrize("n,nfe", [(12801, 700), (20011, 20011)])
def test_crowded_ball(gi, orc, torch_cuda, n, nfe):
    """A remnant's density (600 bodies in a cell): each pair to about 1e-7, as in
    ordinary states."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    pos, _, _ = gi.ic_uniform_ball(n, n, (n / 2500.0) ** (1 / 3))
    run = wl.run_desc(gi, 0, n, nfe)
    ctx = gi.Context(0)
    got = ctx.potential(_dev(torch, pos).data_ptr(), [run], p)[0]
    ctx.close()
    want = orc.potential_fp64(pos, [run], p).sum() / 2.0
    assert abs(got - want) <= 2e-7 * abs(want)


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


def test_workspace_of_large_runs(gi, torch_cuda):
    """Runs whose warps take several tasks each: every pair once (all bodies in one
    point; a task is 4e-6 of the sum), the same bits alone and in a batch, and a
    workspace that does not grow with n^2 (1.15M bodies have 5.1M tasks, 41 MB of
    partial sums at one each)."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    n, nfe, big = 265011, 7000, 1153434
    pos = np.zeros((big, 4), np.float32)
    pos[n:, :3] = np.random.default_rng(3).uniform(-75, 75, size=(big - n, 3))
    d = _dev(torch, pos)
    ctx = gi.Context(0)
    ctx.potential(d.data_ptr(), [wl.run_desc(gi, 0, 20000, 100)], p)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    runs = [wl.run_desc(gi, 0, n, nfe), wl.run_desc(gi, n, big - n, 5)]
    both = ctx.potential(d.data_ptr(), runs, p)
    ctx.potential(d.data_ptr(), [wl.run_desc(gi, 0, big, 31000)], p)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= 8 << 20
    assert ctx.potential(d.data_ptr(), runs[:1], p)[0] == both[0]
    assert ctx.potential(d.data_ptr(), runs[1:], p)[0] == both[1]
    ctx.close()
    want, tol = _coincident(wl, n, nfe)
    assert abs(both[0] - want) <= tol
