"""Batches in two phases (parallel walk into hit lists, then the adds) against
the oracle: one point to several thousand, rows through shared memory (few
points) and through registers, row widths around the column layouts, points of
no, one and many hits, several states, a list per (point, node) and lists from
a common pool, a pool that runs out, and FP32C, whose lists hold only the
terms it keeps."""
import itertools

import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu
FP32C_TOL = 1e-7


def _run(g, X, precision=H.FP64, counts=None):
    import torch
    return H.interpolate(g, torch.from_numpy(X).cuda(), counts=counts, precision=precision).cpu().numpy()


@pytest.mark.parametrize("td", [1, 32, 33, 64, 118, 257])
@pytest.mark.parametrize("npts", [1, 3, 200, 1185, 2500])
def test_every_batch_size_and_width(cuda, npts, td):
    hg = H.HostGrid.adaptive(20, 2600, td, seed=td)
    X = H.gen_points(20, npts, kind=2, seed=npts)
    if npts > 2:
        X[npts // 2, 3] = np.inf
    g = H.Grid(hg, flags=H.BUILD_FP32)
    out, ref = _run(g, X), O.Gold(*hg.arrays()).interpolate(X, nthreads=4)
    ok = np.isfinite(X).all(axis=1)
    assert np.isnan(out[~ok]).all()
    assert np.array_equal(out[ok], ref[ok])
    out32 = _run(g, X, H.FP32C)
    assert np.isnan(out32[~ok]).all()
    assert O.rel_error(out32[ok], ref[ok])[0] <= FP32C_TOL


@pytest.mark.parametrize("counts", [(1, 1, 1), (0, 5, 0), (400, 1, 900)])
def test_states_of_uneven_size(cuda, counts):
    hosts = [H.HostGrid.adaptive(12, n, 40, seed=n) for n in (1, 130, 9000)]
    grids = [H.Grid(h) for h in hosts]
    X = H.gen_points(12, sum(counts), kind=2, seed=3)
    out = _run(grids, X, counts=list(counts))
    at = 0
    for h, c in zip(hosts, counts):
        if c:
            assert np.array_equal(out[at:at + c], O.Gold(*h.arrays()).interpolate(X[at:at + c], nthreads=4))
        at += c


def test_many_hits_in_one_walk_chunk(cuda):
    """A regular grid: hundreds of hits per walk chunk, past the warp's list."""
    hg = H.HostGrid.regular(10, 5, 24, seed=1)
    X = H.gen_points(10, 3000, kind=0, seed=2)
    g, ref = H.Grid(hg), O.Gold(*hg.arrays())
    for n in (1, 90, 3000):
        assert np.array_equal(_run(g, X[:n]), ref.interpolate(X[:n], nthreads=4)), n


@pytest.mark.parametrize("npts,nno,td", [(1900, 3000, 33), (1900, 3000, 64), (145, 15_000, 40)])
def test_pool_that_runs_out(cuda, npts, nno, td):
    """Every node is narrow in three of 48 dimensions, so that uniform points
    hardly ever meet one and the pool is sized for few hits; points in the
    middle meet them all and need more entries than it has.  The points that
    find none are walked again."""
    rng = np.random.default_rng(4)
    dims = np.array(list(itertools.islice(itertools.combinations(range(48), 3), nno - 1)))
    idx = np.zeros((nno, 96), np.int32)
    rows = np.arange(1, nno)[:, None]
    idx[rows, dims], idx[rows, 48 + dims] = 64, 31
    sur = rng.standard_normal((nno, td))
    X = np.full((npts, 48), 31 / 64) + rng.uniform(-0.5, 0.5, (npts, 48)) / 64
    X[0] = 0.9
    g = H.Grid(H.HostGrid.from_dense(idx, sur))
    assert np.array_equal(_run(g, X), O.Gold(idx, sur).interpolate(X, nthreads=4))


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("td", [20, 33, 64, 65, 118, 128])
def test_fp32c_big_term_lists(cuda, td, variant):
    """Narrow rows list their big terms: points of no, a few and hundreds of
    big terms (surpluses that do not decay with the level make every term
    big), whole and short groups, against the oracle."""
    idx, sur = H.HostGrid.adaptive(14, 3000, td, seed=td).arrays()
    X = H.gen_points(14, 1500, kind=2, seed=3)
    prev = H.set_fp32c_variant(variant)
    try:
        for s in (sur, np.sign(sur) * (0.5 + np.abs(sur) / (1 + np.abs(sur).max()))):
            g = H.Grid(H.HostGrid.from_dense(idx, s), flags=H.BUILD_FP32)
            err = O.rel_error(_run(g, X, H.FP32C), O.Gold(idx, s).interpolate(X, nthreads=4))[0]
            assert err <= FP32C_TOL
    finally:
        H.set_fp32c_variant(prev)
