"""Small FP64 host calls whose points and values each fit the pinned staging
buffers are copied by the call's graph; larger ones are copied around it.
Both sides of the limit, alternating, on one grid and from two threads."""
import threading

import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu


def test_staged_and_unstaged_calls_alternate(cuda):
    hg = H.HostGrid.adaptive(10, 2000, 64, seed=5)
    g, gold = H.Grid(hg), O.Gold(*hg.arrays())
    X = H.gen_points(10, 256, kind=2, seed=6)
    ref = gold.interpolate(X)
    for n in (128, 129, 1, 256, 128, 129, 1):     # 128 points of 64 values are 64 KB
        assert np.array_equal(H.interpolate_host(g, X[:n]), ref[:n]), n


def test_staged_calls_from_two_threads(cuda):
    hg = H.HostGrid.adaptive(10, 2000, 24, seed=7)
    g = H.Grid(hg)
    X = H.gen_points(10, 40, kind=2, seed=8)
    ref = O.Gold(*hg.arrays()).interpolate(X)
    bad = []

    def work(k):
        for r in range(30):
            p = (7 * k + r) % 40
            if not np.array_equal(H.interpolate_host(g, X[p:p + 1])[0], ref[p]):
                bad.append((k, r))

    t = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [th.start() for th in t]
    [th.join() for th in t]
    assert not bad
