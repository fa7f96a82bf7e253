"""FP64 form on batches above the small-batch size: hits are listed and their
weights and rows taken 32 at a time, the rows in groups that fill a lane's
registers whatever the row width.  Checked bit for bit against the oracle at
the row widths where the column layout changes, on grids whose points have
fewer hits than one list, about one list, and many."""
import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("td", [1, 31, 32, 33, 64, 65, 118, 128, 129, 256, 257])
@pytest.mark.parametrize("dim,nno", [(3, 5), (10, 60), (30, 3000)])
def test_fp64_rows_of_every_width_match_oracle(cuda, dim, nno, td):
    import torch
    hg = H.HostGrid.adaptive(dim, nno, td, seed=td + dim)
    X = H.gen_points(dim, 1300, kind=2, seed=7)
    X[17, 1] = np.nan
    g = H.Grid(hg)
    out = H.interpolate(g, torch.from_numpy(X).cuda()).cpu().numpy()
    ref = O.Gold(*hg.arrays()).interpolate(X, nthreads=4)
    assert np.isnan(out[17]).all()
    keep = np.arange(len(X)) != 17
    assert np.array_equal(out[keep], ref[keep])


@pytest.mark.parametrize("rows", [32, 33, 1000])
def test_fp64_lists_carry_across_node_chunks(cuda, rows):
    import torch
    hg = H.HostGrid.adaptive(30, 3000, 70, seed=5)
    X = H.gen_points(30, 1300, kind=2, seed=8)
    g = H.Grid(hg)
    prev = H.set_chunk_rows(rows)
    try:
        out = H.interpolate(g, torch.from_numpy(X).cuda()).cpu().numpy()
    finally:
        H.set_chunk_rows(prev)
    assert np.array_equal(out, O.Gold(*hg.arrays()).interpolate(X, nthreads=4))
