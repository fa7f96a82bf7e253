"""Batches in two phases, each way the dispatch has through them, with the way
that ran read from the launch statistics: rows through shared memory (blocks of
128 threads) or registers (256), several states at once, more walk chunks than
a block takes at a time, and a pool of list entries that runs out on either
way, bit for bit against the oracle; and batches around one heavy point, which
must fit the pool."""
import ctypes
import itertools

import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu
STAGED, GATHERED = 128, 256


def _check(grids, X, golds, counts, threads):
    import torch
    out = H.interpolate(grids, torch.from_numpy(X).cuda(), counts=counts).cpu().numpy()
    s = H.last_launch()
    assert (s.kernels, s.block_threads) == (2, threads)
    at = 0
    for gold, c in zip(golds, counts):
        if c:
            ok = np.isfinite(X[at:at + c]).all(axis=1)
            ref = gold.interpolate(X[at:at + c][ok], nthreads=4)
            assert np.array_equal(out[at:at + c][ok], ref) and np.isnan(out[at:at + c][~ok]).all()
        at += c


@pytest.mark.parametrize("counts,nodes,td,threads", [
    ((900,), (2600,), 65, GATHERED), ((900,), (2600,), 118, GATHERED), ((950,), (2600,), 64, GATHERED),
    ((400, 1, 600), (1, 130, 9000), 118, GATHERED), ((0, 500, 0, 501), (50, 3000, 9, 12_000), 66, GATHERED),
    ((3, 0, 40), (1, 130, 9000), 33, STAGED),
    ((1,), (140_000,), 3, STAGED), ((1, 2), (140_000, 135_000), 2, STAGED)])     # more than 1,024 chunks a point
def test_states_and_widths(cuda, counts, nodes, td, threads):
    hosts = [H.HostGrid.adaptive(20, n, td, seed=n) for n in nodes]
    X = H.gen_points(20, sum(counts), kind=2, seed=3)
    if len(X) > 100:
        X[57, 3] = np.nan
    _check([H.Grid(h) for h in hosts], X, [O.Gold(*h.arrays()) for h in hosts], list(counts), threads)


def test_narrow_rows_through_registers(cuda):
    """Grids whose points have hundreds of hits keep the two phases for a few
    thousand points."""
    hosts = [H.HostGrid.adaptive(45, 100_000, 24, seed=s) for s in (5, 6)]
    X = H.gen_points(45, 1810, kind=0, seed=2)
    _check([H.Grid(h) for h in hosts], X, [O.Gold(*h.arrays()) for h in hosts], [900, 910], GATHERED)


@pytest.mark.parametrize("npts,wide,narrow,td,threads", [
    (1100, 0, 3000, 64, GATHERED), (1100, 0, 3000, 118, GATHERED), (1900, 1000, 17_000, 5, GATHERED),
    (250, 0, 15_000, 40, STAGED)])
def test_pool_that_runs_out(cuda, npts, wide, narrow, td, threads):
    """`narrow` nodes are narrow in three of 48 dimensions, so that uniform
    points hardly ever meet one and the pool is sized for the `wide` ones,
    active everywhere; the points in the middle meet them all.  The points that
    find no room are walked again, one without a hit and one with a coordinate
    that is not finite among them."""
    rng = np.random.default_rng(4)
    idx = np.zeros((1 + wide + narrow, 96), np.int32)
    for k, pair in enumerate(itertools.islice(itertools.combinations(range(48), 2), wide)):
        idx[1 + k, list(pair)] = 1                # hats 1 - x
    for k, dims in enumerate(itertools.islice(itertools.combinations(range(48), 3), narrow)):
        d = np.array(dims)
        idx[1 + wide + k, d], idx[1 + wide + k, 48 + d] = 64, 31
    sur = rng.standard_normal((len(idx), td))
    X = np.full((npts, 48), 31 / 64) + rng.uniform(-0.5, 0.5, (npts, 48)) / 64
    X[-1], X[-2, 7] = 0.9, np.nan
    # the lists hold at most max(2.5 M, 16 entries per point and wide node)
    assert (npts - 2) * len(idx) > min(max(2.5 * 2 ** 20, 16 * npts * (wide + 2)), (256 << 20) / 12)
    _check([H.Grid(H.HostGrid.from_dense(idx, sur))], X, [O.Gold(idx, sur)], [npts], threads)


def test_batch_around_a_heavy_point(cuda):
    """300 points around the one with the most active nodes of 4,000 take no
    longer than by the one-phase kernels (sgi_interpolate_noalloc); when their
    hits did not fit the pool they took more than twice as long."""
    import torch
    g = H.Grid(H.HostGrid.adaptive(59, 150_000, 118, seed=5))
    cloud = torch.from_numpy(H.gen_points(59, 4000, kind=0, seed=1)).cuda()
    n = H.active_count(g, cloud)
    heavy = cloud[int(n.argmax())]
    x = (heavy + 1e-4 * torch.from_numpy(np.random.default_rng(1).standard_normal((300, 59))).cuda()).clamp_(0, 1)
    out = torch.empty((300, 118), dtype=torch.float64, device="cuda")
    offs = np.array([0, 300], np.int64)
    f = H.lib.sgi_interpolate_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                  ctypes.c_void_p]
    arr = (ctypes.c_void_p * 1)(g.handle.value)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    res = {}

    def one_phase():
        assert f(1, arr, offs.ctypes.data, x.data_ptr(), out.data_ptr(), H.FP64, stream) == 0

    def two_phase():
        res["out"] = H.interpolate(g, x)
        assert H.last_launch().kernels == 2

    def best(call):
        times = []
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            call()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    t1, t2 = best(one_phase), best(two_phase)
    assert torch.equal(res["out"], out)
    assert t2 <= t1, (t1, t2)
