"""The contact pass's grid builds (none, one cluster per run, grid-wide) and
the far field's splits of short runs, at the run sizes where the library
changes from one to the next: a run's forces are the same bits alone and
beside a run that takes the grid-wide build, and match the FP64 oracle."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _aliased(seed, n):
    """Bodies whose cells meet on the torus of buckets: a crowded clump, copies
    of its cells whole torus widths away (16 to 256 cells, each axis), singles
    strewn over the aliases, and bodies at the cells' range limits."""
    rng = np.random.default_rng(seed)
    pos = np.zeros((n, 4), np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    x = d * 2.2 * rng.uniform(size=(n, 1)) ** 0.6
    part = rng.uniform(size=n)
    far = part > 0.6
    shift = rng.choice([-256, -64, -32, -16, 0, 16, 32, 64, 128], size=(n, 3))
    x[far] += shift[far]
    gas = part > 0.8  # sparse elsewhere, so that the oracle's sums stay plain
    x[gas] = rng.uniform(-60, 60, size=(gas.sum(), 3))
    pos[:, :3] = x
    pos[:3, :3] = [[3e9, 0, 0], [-3e9, 1, 1], [3e9, 0.25, 0.25]]
    vel = np.zeros((n, 4), np.float32)
    vel[:, :3] = rng.normal(scale=1.5, size=(n, 3))
    return pos, vel


@pytest.mark.parametrize("n", [1, 9, 3072, 3073, 4096, 4097, 6145, 12287, 12288, 32768, 65535, 65536,
                               131071])
def test_sizes_at_path_limits(gi, orc, torch_cuda, n):
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    ctx = gi.Context(0)
    pos, vel = _aliased(n, n) if n > 16 else (np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32))
    pos[:, :3] += np.arange(n)[:, None] * np.float32(1e-3) if n <= 16 else 0
    nfe = n // 7
    big, bvel, bfe = gi.ic_uniform_ball(5, 131072, 60.0)
    run = wl.run_desc(gi, 0, n, nfe)
    dp, dv = _dev(torch, np.concatenate([pos, big])), _dev(torch, np.concatenate([vel, bvel]))
    alone, both = torch.zeros_like(dp), torch.zeros_like(dp)
    ctx.forces(dp.data_ptr(), dv.data_ptr(), alone.data_ptr(), [run], p)
    ctx.forces(dp.data_ptr(), dv.data_ptr(), both.data_ptr(), [run, wl.run_desc(gi, n, 131072, bfe)], p)
    torch.cuda.synchronize()
    assert torch.equal(alone[:n], both[:n])
    idx = np.unique(np.linspace(0, n - 1, 96).astype(np.int32))
    f64, _ = orc.forces_fp64(pos, vel, [run], p, idx=idx)
    got = alone.cpu().numpy()[idx, :3]
    if n > 1:
        assert rel_l2(got, f64) < FORCE_TOL
    else:
        assert not got.any()
    ctx.close()


@pytest.mark.parametrize("n,nfe", [(1, 0), (33, 33), (129, 5), (3000, 0), (12288, 300), (12289, 700), (20011, 20011),
                                   (33000, 1000)])
def test_potential_sizes(gi, orc, torch_cuda, n, nfe):
    """Pair potential at the sizes where its decomposition changes, with the
    Fe boundary inside a lane group, a chunk, at 0 and at n: the FP64 oracle's
    to the FP32 pair arithmetic (each term to about 1e-7), and the same bits
    alone and in a batch."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    pos, vel, _ = gi.ic_uniform_ball(n, n, max(1.0, (n / 4.0) ** (1 / 3)))
    other, ovel, ofe = gi.ic_uniform_ball(77, 15000, 30.0)
    d = _dev(torch, np.concatenate([pos, other]))
    ctx = gi.Context(0)
    run, rest = wl.run_desc(gi, 0, n, nfe), wl.run_desc(gi, n, 15000, ofe)
    alone = ctx.potential(d.data_ptr(), [run], p)[0]
    both = ctx.potential(d.data_ptr(), [rest, run], p)
    assert both[1] == alone and ctx.potential(d.data_ptr(), [rest], p)[0] == both[0]
    want = orc.potential_fp64(pos, [run], p).sum() / 2.0
    assert abs(alone - want) <= 2e-7 * abs(want)
    ctx.close()


@pytest.mark.parametrize("m", [31, 32, 33, 64, 95, 127, 128, 129, 160, 257, 700])
@pytest.mark.parametrize("spread", [0.3, 0.99])
def test_crowded_cell_sizes(gi, torch_cuda, m, spread):
    """Neighbouring cells of m bodies each, at the sizes where the tiled path's
    chunks, staged blocks and tiles end, packed (all pairs are contacts) or
    over their cells (few are), bodies alone beside them and a coincident
    pair: the same bits tiled and on the row path."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    rng = np.random.default_rng(1000 * m + int(100 * spread))
    cells = np.array([(0, 0, 0), (1, 0, 0), (1, 1, 0), (-1, 0, 1), (0, -1, -1)], np.float64)
    n = 5 * m + 4000
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    x = rng.uniform(-9, 9, size=(n, 3))
    for k, c in enumerate(cells):
        x[k * m:(k + 1) * m] = c + rng.uniform(0, spread, size=(m, 3))
    x[5 * m:5 * m + 40] = rng.uniform(-2, 3, size=(40, 3))
    x[1] = x[0]
    x = x[rng.permutation(n)]  # the Fe boundary falls inside the cells
    pos[:, :3] = x
    vel[:, :3] = rng.normal(scale=1.5, size=(n, 3))
    run = wl.run_desc(gi, 0, n, n // 3)
    dp, dv = _dev(torch, pos), _dev(torch, vel)
    out = []
    for dense_min in (32, 1 << 30):
        ctx = gi.Context(0, dense_min=dense_min)
        f = torch.zeros_like(dp)
        ctx.forces(dp.data_ptr(), dv.data_ptr(), f.data_ptr(), [run], p)
        torch.cuda.synchronize()
        out.append(f)
        ctx.close()
    assert torch.equal(out[0], out[1])


def test_calls_after_one_another(gi, torch_cuda):
    """The far-field sums are left clean for the next call on the stream: a
    run's forces are a fresh context's, after larger and smaller runs, runs
    with bodies between them, one-sided calls and graphs of either kind."""
    import gi_workloads as wl
    torch = torch_cuda
    p = wl.params(gi)
    sizes = [(20000, 0), (700, 0), (5000, 300), (33000, 7), (1, 0), (9000, 20000)]
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        s = st.cuda_stream
        pos, vel = _aliased(3, 42000)
        dp, dv = _dev(torch, pos), _dev(torch, vel)
        state = [t.clone() for t in (dp, dv, dp, dv)]
        ctx = gi.Context(0)

        def force(c, n, off):
            f = torch.zeros_like(dp)
            c.forces(dp.data_ptr(), dv.data_ptr(), f.data_ptr(), [wl.run_desc(gi, off, n, n // 5)], p, s)
            st.synchronize()
            return f

        def graph(n):
            q = [t.data_ptr() for t in state]
            return ctx.graph(*q, [wl.run_desc(gi, 0, n, n // 5)], p, 3, s)

        want = []
        for n, off in sizes:
            c = gi.Context(0)
            want.append(force(c, n, off))
            c.close()
        force(ctx, 42000, 0)  # a graph keeps the scratch it was captured with: no call may outgrow it
        graphs = [graph(30000)]
        for rep in range(3):
            for (n, off), w in zip(sizes, want):
                assert torch.equal(force(ctx, n, off), w)
                for g in graphs:
                    g.launch(s)
            if rep == 0:
                ctx.set_options(accum=gi.GI_ACCUM_FP64)
                force(ctx, 25000, 0)
                graphs.append(graph(12000))
                ctx.set_options()
        for g in graphs:
            g.close()
        ctx.close()
