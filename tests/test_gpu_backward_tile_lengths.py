"""The backward's tiles of sorted pairs take their length from the number of
pairs (32 to 1,024): nodes that begin before a tile, cover it and go on after
it, at every length, many more than 32 tiles of one node, tiles in which nearly
every pair begins a node, odd and even row widths.  Against the oracle's
gradient (tolerances of the other gradient tests), and either gradient alone bit for bit against both."""
import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nno,npts,td", [
    (2, 1, 2048, 3), (2, 1, 131_073, 40),          # one node, 64 and 4,097 tiles of 32
    (3, 5, 2049, 70), (3, 9, 3100, 118), (3, 9, 40_000, 33),
    (2, 9, 1_200_000, 2),                          # tiles of 1,024
    (10, 3000, 300, 8), (10, 3000, 300, 63), (10, 3000, 300, 117), (10, 3000, 300, 118), (10, 3000, 40, 256),
    (20, 2000, 12_000, 5)])
def test_backward_at_every_tile_length(cuda, dim, nno, npts, td):
    import torch
    hg = H.HostGrid.adaptive(dim, nno, td, seed=dim + td)
    X = H.gen_points(dim, npts, kind=0, seed=1, kink_reject=1e-6)
    C = np.random.default_rng(2).standard_normal((npts, td))
    g = H.Grid(hg)
    x, c = torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda()
    gx, gs = H.backward(g, x, c)
    ox, os_ = O.Gold(*hg.arrays()).gradient(X, C)
    assert np.abs(gx.cpu().numpy() - ox).max() <= 1e-10 * (np.abs(ox).max() + 1e-300)
    # sums of n terms of either sign in two orders: rounding errors of about
    # n 2^-53 of a term (1.3e-10 at 1.2 million points), where the largest
    # sums are sqrt(n) terms
    assert np.abs(gs.cpu().numpy() - os_).max() <= 1e-12 * (np.abs(os_).max() + 1e-300)
    assert torch.equal(H.backward(g, x, c, want_surplus=False)[0], gx)
    assert torch.equal(H.backward(g, x, c, want_x=False)[1], gs)


@pytest.mark.parametrize("want_x", [True, False])
def test_small_batch_spreads_over_the_gpu(cuda, want_x):
    """A few hundred points: at most 64 pairs per warp of the node pass (with
    1,024 it took 33 warps and twelve times as long)."""
    import torch
    hg = H.HostGrid.adaptive(59, 4000, 64, seed=3)
    x = torch.from_numpy(H.gen_points(59, 256, kind=2, seed=1)).cuda()
    g = H.Grid(hg)
    pairs = int(H.active_count(g, x).sum())
    H.backward(g, x, torch.ones((256, 64), dtype=torch.float64, device="cuda"), want_x=want_x)
    s = H.last_launch()
    assert s.grid_blocks * s.block_threads // 32 * 64 >= pairs
