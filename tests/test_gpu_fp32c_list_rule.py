"""FP32C descent kernels with and without the list of big terms, which a launch
takes by its grids' mean active nodes (100 and more list them; of few points,
where that times the root of their share of the nodes is 16 and more): a grid
on either side and both in one call, every variant, row widths around the column
layouts, whole grids and node chunks, surpluses whose big terms are few and
surpluses that make every term big."""
import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu
FP32C_TOL = 1e-7


def _mean_active(idx):
    """Sum over the nodes of their supports' share of the unit cube."""
    dim = idx.shape[1] // 2
    i, j = idx[:, :dim].astype(float), idx[:, dim:].astype(float)
    length = np.maximum(0, np.minimum(i, j + 1) - np.maximum(0, j - 1)) / np.maximum(i, 1)
    return np.where(i > 0, length, 1.0).prod(axis=1).sum()


def _hosts(td, flat):
    for nno, lists in ((12_000, True), (1500, False)):
        idx, sur = H.HostGrid.adaptive(30, nno, td, seed=6).arrays()
        a = _mean_active(idx)
        assert (a >= 110 and a * np.sqrt(a / nno) >= 17) if lists else (a <= 90)
        if flat:
            sur = np.sign(sur) * (0.5 + np.abs(sur) / (1 + np.abs(sur).max()))
        yield idx, sur


@pytest.mark.parametrize("rows", [-1, 1000])
@pytest.mark.parametrize("variant", [0, 1, 2, H.FP32C_AUTO])
@pytest.mark.parametrize("td", [20, 33, 64, 65, 118, 128, 200])
def test_both_sides_of_the_line(cuda, td, variant, rows):
    import torch
    X = H.gen_points(30, 1300, kind=2, seed=3)
    x = torch.from_numpy(np.concatenate([X, X[:500]])).cuda()
    prev, prev_v = H.set_chunk_rows(rows), H.set_fp32c_variant(variant)
    try:
        for flat in (False, True):
            hosts = list(_hosts(td, flat))
            grids = [H.Grid(H.HostGrid.from_dense(*h), flags=H.BUILD_FP32) for h in hosts]
            refs = [O.Gold(*h).interpolate(X, nthreads=4) for h in hosts]
            for g, ref in zip(grids, refs):
                got = H.interpolate(g, x[:1300], precision=H.FP32C).cpu().numpy()
                assert O.rel_error(got, ref)[0] <= FP32C_TOL
            got = H.interpolate(grids, x, counts=[1300, 500], precision=H.FP32C).cpu().numpy()
            assert O.rel_error(got, np.concatenate([refs[0], refs[1][:500]]))[0] <= FP32C_TOL
    finally:
        H.set_chunk_rows(prev)
        H.set_fp32c_variant(prev_v)
