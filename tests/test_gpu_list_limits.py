"""Batches in two phases at the limits of their scratch: calls whose lists
would not fit it run on the one-phase kernels, with the same bits."""
import itertools
import subprocess
import sys

import numpy as np
import pytest

import hddm_b200 as H
import oracle as O
from conftest import PKG, ROOT

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
    sur = np.random.default_rng(1).standard_normal((len(idx), 130))
    X = np.random.default_rng(2).uniform(0.02, 0.98, (8192, 10))
    out = H.interpolate(H.Grid(H.HostGrid.from_dense(idx, sur)), torch.from_numpy(X).cuda()).cpu().numpy()
    assert H.last_launch().kernels == 1
    some = [0, 1, 4095, 8000, 8191]
    assert np.array_equal(out[some], O.Gold(idx, sur).interpolate(X[some], nthreads=4))


SCRIPT = r"""
import sys
sys.path[:0] = [{root!r}, {pkg!r}]
import numpy as np
import torch
import hddm_b200 as H
import oracle as O
hg = H.HostGrid.adaptive(30, 100_000, 8, seed=1)
X = H.gen_points(30, 2000, kind=0, seed=2)
g, x = H.Grid(hg), torch.from_numpy(X).cuda()
out = torch.zeros((2000, 8), dtype=torch.float64, device="cuda")
plan = H.Plan(g, x, out, chunk_rows=0)
assert plan.launches == 2
two = plan.launch().clone()
one = torch.zeros_like(out)
del plan
fill = torch.empty(torch.cuda.mem_get_info()[0] - (160 << 20), dtype=torch.uint8, device="cuda")
plan = H.Plan(g, x, one, chunk_rows=0)
assert plan.launches == 1, plan.launches
plan.launch()
torch.cuda.synchronize()
del fill, plan
assert torch.equal(one, two)
assert np.array_equal(one[:200].cpu().numpy(), O.Gold(*hg.arrays()).interpolate(X[:200], nthreads=4))
"""


def test_plan_without_room_for_its_lists(cuda):
    """A plan whose list scratch (more than 200 MB here) finds no room on the
    device records the one-phase kernels instead of failing.  In a child
    process: device memory that the library's pool kept would make room."""
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT, pkg=PKG)], timeout=180, capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr[-2000:]
