"""Batches in two phases at the limits of their scratch: calls whose lists
would not fit it run on the one-phase kernels, with the same bits."""
import itertools

import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu


def test_more_chunks_than_the_scratch_holds(cuda):
    """8,192 points of 778,240 nodes, a third of them active everywhere and the
    others on half of the cube: 50 million chunks of 128 nodes, whose table
    alone is larger than the scratch, and more entries than 32 bits number."""
    import torch
    const, left, right, tent = (0, 0), (1, 0), (1, 1), (2, 1)
    opts = np.array([const, left, right, tent], np.int32)
    last = np.array([(4, 1), (4, 3), tent], np.int32)
    pick = np.array(list(itertools.product(range(4), repeat=9)))          # 4^9 rows
    idx = np.zeros((3 * len(pick), 20), np.int32)
    for d in range(9):
        pair = np.repeat(opts[pick[:, d]], 3, axis=0)
        idx[:, d], idx[:, 10 + d] = pair[:, 0], pair[:, 1]
    idx[:, 9], idx[:, 19] = np.tile(last[:, 0], len(pick)), np.tile(last[:, 1], len(pick))
    idx = idx[:95 * 8192]
    sur = np.random.default_rng(1).standard_normal((len(idx), 1))
    X = np.random.default_rng(2).uniform(0.02, 0.98, (8192, 10))
    out = H.interpolate(H.Grid(H.HostGrid.from_dense(idx, sur)), torch.from_numpy(X).cuda()).cpu().numpy()
    assert H.last_launch().kernels == 1
    some = [0, 1, 4095, 8000, 8191]
    assert np.array_equal(out[some], O.Gold(idx, sur).interpolate(X[some], nthreads=4))
