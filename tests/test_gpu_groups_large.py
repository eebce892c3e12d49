"""Grouping at the sizes where the cell table outgrows L2 and the sparse link kernels
take over, against connected components of the touching pairs (k-d tree, each pair
decided by the reference's FP32 test)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOUCH = 1.5


def _components(pos):
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    from scipy.spatial import cKDTree
    n = len(pos)
    x = pos[:, :3]
    pairs = cKDTree(x.astype(np.float64)).query_pairs(TOUCH * (1 + 1e-5), output_type="ndarray")
    d = x[pairs[:, 0]] - x[pairs[:, 1]]
    sq = d * d
    r2 = (sq[:, 0] + sq[:, 1]) + sq[:, 2]
    pairs = pairs[np.sqrt(r2) < np.float32(TOUCH)]
    g = coo_matrix((np.ones(len(pairs), np.int8), (pairs[:, 0], pairs[:, 1])), shape=(n, n))
    k, label = connected_components(g, directed=False)
    first = np.full(k, n, np.int64)
    np.minimum.at(first, label, np.arange(n))
    return first[label]


def _ball(rng, n, rho):
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return d * (3 * n / (4 * np.pi * rho)) ** (1 / 3) * rng.uniform(size=(n, 1)) ** (1 / 3)


@pytest.mark.parametrize("n", [149999, 150000, 262145])
@pytest.mark.parametrize("state", ["gas", "raw", "mixed"])
def test_groups_of_many_bodies(gi, torch_cuda, n, state):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    if state == "mixed":  # settled and crowded bodies, strings of bodies, gas, bodies without a cell
        x = np.concatenate([_ball(rng, n // 2, 4.3), _ball(rng, n // 8, 300.0) + [80.0, 0, 0],
                            _ball(rng, n - n // 2 - n // 8, 0.02) + [0, 200.0, 0]])
        x[-3000:, 0] = -100.0 - 1.499 * np.arange(3000)
        x[-3000:, 1:] = 0.0
        x[-3010:-3000] = [3e9, 0, 0]
        x = x[rng.permutation(n)]
    else:
        x = _ball(rng, n, 0.1 if state == "gas" else 0.955)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = x
    d = torch.from_numpy(pos).cuda()
    group = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    ctx = gi.Context(0)
    em = gi.find_earth_moon(ctx, d.data_ptr(), n, TOUCH, [n // 5, 2 * n // 5, 3 * n // 5], group.data_ptr())
    ctx.close()
    want = _components(pos)
    assert np.array_equal(group.cpu().numpy(), want)
    sizes = np.bincount(want, minlength=n)
    assert em.n_groups == (sizes > 0).sum() and em.n_earth == sizes.max() and em.earth_label == sizes.argmax()
