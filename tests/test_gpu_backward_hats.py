"""dL/dx multiplies each term by 1 / hat (two Newton-Raphson steps from the
approximate reciprocal): its error over the whole range of hats, [2^-53, 1],
seen through grids of one term, where everything else is exact; and dimensions
whose gradient copies leave room for fewer warps per block."""
import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu


def _both_ways(idx, sur, X, C):
    import torch
    g = H.Grid(H.HostGrid.from_dense(idx, sur))
    x, c = torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda()
    gx, gs = H.backward(g, x, c)
    assert torch.equal(H.backward(g, x, c, want_surplus=False)[0], gx)
    return gx.cpu().numpy(), gs.cpu().numpy()


def test_reciprocal_of_every_hat(cuda):
    """One node of one dimension, i = 2, j = 1, surplus and dL/dvalue 1: the
    weight is the hat h, and dL/dx = fl(2 h r) for r close to 1 / h, so that
    |dL/dx| / 2 - 1 is r's relative error, at most two ulps (2^-51), and one
    rounding (2^-53)."""
    rng = np.random.default_rng(1)
    k = np.unique(np.concatenate([np.arange(1, 2049), 2 ** np.arange(0, 53), 2 ** np.arange(1, 54) - 1,
                                  2 ** 53 - 2 ** np.arange(1, 12),
                                  (2.0 ** rng.uniform(0, 53, 300_000)).astype(np.int64)]))
    k = k[k < 2 ** 53]
    x = np.concatenate([k * 2.0 ** -54, 1.0 - (k[k % 2 == 0] // 2) * 2.0 ** -53])     # left and right of the centre
    h = 1.0 - np.abs(x * 2.0 - 1.0)
    x = x[(h > 0) & (h < 1)]
    h = h[(h > 0) & (h < 1)]
    assert h.min() == 2.0 ** -53 and h.max() > 1 - 2.0 ** -50
    gx, gs = _both_ways(np.array([[2, 1]], np.int32), np.ones((1, 1)), x[:, None], np.ones((len(x), 1)))
    assert np.array_equal(np.sign(gx[:, 0]), np.where(x < 0.5, 1.0, -1.0))
    assert np.abs(np.abs(gx[:, 0]) / 2 - 1).max() <= 2.0 ** -51 + 2.0 ** -53
    assert abs(gs[0, 0] - h.sum()) <= 1e-12 * h.sum()


def test_terms_of_tiny_hats(cuda):
    """Products of three hats down to 2^-50: each gradient within the
    reciprocal's two ulps and seven roundings of the exact product."""
    rng = np.random.default_rng(2)
    X = np.concatenate([2.0 ** -rng.uniform(1.1, 50, (4000, 3)), 1.0 - 2.0 ** -rng.uniform(1.1, 50, (4000, 3))])
    s, c = 1.7, rng.standard_normal((len(X), 1))
    gx, _ = _both_ways(np.array([[2, 2, 2, 1, 1, 1]], np.int32), np.full((1, 1), s), X, c)
    h = (1.0 - np.abs(X * 2.0 - 1.0)).astype(np.longdouble)
    for d in range(3):
        a, b = h[:, (d + 1) % 3], h[:, (d + 2) % 3]
        ref = c[:, 0].astype(np.longdouble) * np.longdouble(s) * a * b * np.where(X[:, d] < 0.5, 2, -2)
        assert (np.abs(gx[:, d] - ref) <= (2.0 ** -51 + 7 * 2.0 ** -53) * np.abs(ref)).all()


@pytest.mark.parametrize("dim", [340, 400, 1800])
def test_dimensions_with_few_warps_per_block(cuda, dim):
    """Eight, six and one warps of bwd_points_kernel per block (1,300 points of
    a few active nodes), and the same through hit lists (100 points)."""
    rng = np.random.default_rng(dim)
    idx = np.zeros((40, 2 * dim), np.int32)
    for n in range(1, 40):
        d = rng.choice(dim, 1 + n % 3, replace=False)
        idx[n, d], idx[n, dim + d] = 4, rng.choice([1, 3], len(d))
    sur = rng.standard_normal((40, 5))
    X, C = rng.uniform(0, 1, (1300, dim)), rng.standard_normal((1300, 5))
    for n in (1300, 100):
        gx, gs = _both_ways(idx, sur, X[:n], C[:n])
        ox, os_ = O.Gold(idx, sur).gradient(X[:n], C[:n])
        assert np.abs(gx - ox).max() <= 1e-10 * np.abs(ox).max()
        assert np.abs(gs - os_).max() <= 1e-12 * np.abs(os_).max()
