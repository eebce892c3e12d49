"""The FP64 diagnostics of a scope do not depend on bodies outside it, and lose
no digits where the run's first body is far from the scope's bodies: a Moon with
the first body in the Earth, and a first body that escaped or ran away, in the
scope and out of it."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import config1_params

pytestmark = pytest.mark.gpu

# Each term r x w about the centre keeps 2^-48 of |r| |w| through four roundings,
# a thread adds two of them and a warp five levels, each to 2^-47: 18 x 2^-48,
# here 32 x 2^-48 = 2^-43 of S = sqrt(sum m r.r  sum m w.w) >= sum m |r| |w|.
# Terms taken about another point may come to 4 S before the pass is repeated.
L_TOL = 4 * 2.0 ** -43


def _want(pos, vel, mass, sel):
    q = np.longdouble
    m, x, v = mass[sel].astype(q), pos[sel, :3].astype(q), vel[sel, :3].astype(q)
    M = m.sum()
    com, vcom = (m[:, None] * x).sum(0) / M, (m[:, None] * v).sum(0) / M
    r, w = x - com, v - vcom
    L = (m[:, None] * np.cross(r, w)).sum(0)
    S = np.sqrt((m * (r * r).sum(1)).sum()) * np.sqrt((m * (w * w).sum(1)).sum())
    return com, vcom, L, S


@pytest.mark.parametrize("far,speed", [(0.0, 0.0), (1e4, 36.0), (1e6, 36.0), (1e9, 1e3), (1e25, 1e20)])
@pytest.mark.parametrize("scope", [0, 1, 2, 3])
@pytest.mark.parametrize("first", [0, 1, 2])
def test_first_body_far_from_scope(gi, torch_cuda, far, speed, scope, first):
    """first: the label of body 0, which lies in the Earth (label 1) or `far` away."""
    torch = torch_cuda
    rng = np.random.default_rng(5)
    n, nm = 20011, 1500
    x = rng.normal(size=(n, 3)) * 9.0
    v = rng.normal(size=(n, 3)) * 0.7 + 0.1 * np.stack([-x[:, 1], x[:, 0], 0 * x[:, 0]], 1)
    moon = slice(9000, 9000 + nm)
    x[moon] = x[moon] / 5.0 + [360.0, 10.0, -5.0]
    v[moon] += [3.0, 36.0, 1.0]
    label = np.ones(n, np.uint8)
    label[moon] = 2
    label[::7] = 0
    label[0] = first
    if far:
        x[0] = np.array([0.6, -0.64, 0.48]) * far
        v[0] = np.array([-0.36, 0.48, 0.8]) * speed
    sel = [np.ones(n, bool), label > 0, label == 1, label == 2][scope]
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3], vel[:, :3] = x, v
    nfe = 3000
    p = config1_params(gi)
    mass = np.where(np.arange(n) < nfe, p.MassFe, p.MassSi).astype(np.float64)
    run = gi.Run(0, n, nfe, 0, 0, 0, 0, 0)
    dp, dv, dl = (torch.from_numpy(a).cuda() for a in (pos, vel, label))
    ctx = gi.Context(0)
    got = np.array(ctx.diag(dp.data_ptr(), dv.data_ptr(), run, p, dl.data_ptr(), scope))
    ctx.close()
    com, vcom, L, S = _want(pos, vel, mass, sel)
    if far > 1e18 and sel[0]:
        return  # its own |r| |w| is beyond FP32: no finite sum
    assert got[14] == sel.sum()
    assert np.abs(got[1:4] - com).max() <= 1e-13 * np.abs(pos[sel, :3]).max()
    assert np.abs(got[4:7] - vcom).max() <= 1e-13 * np.abs(vel[sel, :3]).max()
    err = float(np.abs(got[7:10] - L).max() / S)
    print(f"scope {scope}, first body {first} at {far:g}: |error of L| {err:.2e} S")
    assert err <= L_TOL
