"""Backward kernels at the edges of their tiles: the pairs sorted by node are
cut every 1,024 (nodes that begin, end or span several tiles, tiles of one
node, a last tile of a few pairs), lists of 32 hits, row widths around the
lane layout, one or two pairs per list, both gradients or either, against the
oracle's gradient (tolerances of the other gradient tests) and, for either
gradient alone, bit for bit against both."""
import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("td", [1, 31, 33, 64, 65, 118, 129, 256])
@pytest.mark.parametrize("dim,nno,npts", [(3, 5, 3), (2, 1, 1024), (3, 9, 1500), (10, 300, 700), (30, 3000, 257)])
def test_backward_tiles(cuda, dim, nno, npts, td):
    import torch
    hg = H.HostGrid.adaptive(dim, nno, td, seed=dim + td)
    X = H.gen_points(dim, npts, kind=0, seed=1, kink_reject=1e-6)
    C = np.random.default_rng(2).standard_normal((npts, td))
    g = H.Grid(hg)
    x, c = torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda()
    gx, gs = H.backward(g, x, c)
    ox, os_ = O.Gold(*hg.arrays()).gradient(X, C)
    assert np.abs(gx.cpu().numpy() - ox).max() <= 1e-10 * (np.abs(ox).max() + 1e-300)
    assert np.abs(gs.cpu().numpy() - os_).max() <= 1e-12 * (np.abs(os_).max() + 1e-300)
    assert torch.equal(H.backward(g, x, c, want_surplus=False)[0], gx)
    assert torch.equal(H.backward(g, x, c, want_x=False)[1], gs)


def test_backward_point_outside_every_support(cuda):
    """A NaN coordinate leaves its nodes inactive; the others still count, in
    both entry forms, and no other point's gradient changes."""
    import torch
    hg = H.HostGrid.adaptive(10, 500, 40, seed=3)
    X = H.gen_points(10, 100, kind=0, seed=4, kink_reject=1e-6)
    C = np.random.default_rng(5).standard_normal((100, 40))
    g = H.Grid(hg)
    ref = H.backward(g, torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda())[0]
    X[31, 2] = np.nan
    x, c = torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda()
    gx, gs = H.backward(g, x, c)
    only = H.backward(g, x, c, want_surplus=False)[0]
    assert torch.equal(gx, only) and bool(torch.isfinite(gx).all()) and bool(torch.isfinite(gs).all())
    keep = torch.arange(100, device="cuda") != 31
    assert torch.equal(gx[keep], ref[keep])


def test_nan_gout_at_hat_centres(cuda):
    """A NaN in dL/dvalue reaches dL/dx also where the slope is 0: at the
    origin every active non-constant hat is at its centre.  NaN in the same
    places as in the oracle, in both entry forms."""
    import torch
    hg = H.HostGrid.adaptive(10, 500, 40, seed=3)
    X = H.gen_points(10, 100, kind=0, seed=4, kink_reject=1e-6)
    X[7] = 0.0
    C = np.random.default_rng(5).standard_normal((100, 40))
    C[[7, 8], [3, 39]] = np.nan
    ox = O.Gold(*hg.arrays()).gradient(X, C)[0]
    assert np.isnan(ox[7]).any()
    g = H.Grid(hg)
    x, c = torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda()
    for want in (True, False):
        gx = H.backward(g, x, c, want_surplus=want)[0].cpu().numpy()
        assert np.array_equal(np.isnan(gx), np.isnan(ox))


@pytest.mark.parametrize("npts,nno", [(200, 3000), (145, 15_000)])
def test_dx_alone_through_lists(cuda, npts, nno):
    """dL/dx alone on a small batch is added from hit lists; here every node is
    narrow in three of 48 dimensions, so that the lists' pool is sized for few
    hits, and the points in the middle meet all nodes: the larger batch runs
    out of room.  Either way the bits are those of both gradients' kernels."""
    import itertools

    import torch
    rng = np.random.default_rng(4)
    dims = np.array(list(itertools.islice(itertools.combinations(range(48), 3), nno - 1)))
    idx = np.zeros((nno, 96), np.int32)
    rows = np.arange(1, nno)[:, None]
    idx[rows, dims], idx[rows, 48 + dims] = 64, 31
    g = H.Grid(H.HostGrid.from_dense(idx, rng.standard_normal((nno, 40))))
    X = np.full((npts, 48), 31 / 64) + rng.uniform(-0.5, 0.5, (npts, 48)) / 64
    X[0], X[5, 7] = 0.9, np.nan
    x = torch.from_numpy(X).cuda()
    c = torch.from_numpy(rng.standard_normal((npts, 40))).cuda()
    assert torch.equal(H.backward(g, x, c, want_surplus=False)[0], H.backward(g, x, c)[0])
