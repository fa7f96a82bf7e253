"""The calls whose speed is measured, and how their inputs are made.

A case is one call of the framework's Python interface on grids and points of
the kinds that the tests and the benchmark use: adaptive grids (refined at
random from the root, levels up to 7, in 10 to 59 dimensions, 10,000 to
300,000 nodes) and regular ones, TotalDof from 8 to 256 (118 is the solver's
own), and from one point per call to a quarter of a million.

  call   "host"    interpolate_host: host arrays in and out (the solver's plugin call)
         "device"  interpolate: device tensors, one grid or a multistate set
         "grad"    backward: gradients for the points, or for points and surpluses
  form   "fp64" or "fp32c"
  states, nodes, nodes_last    node counts of the states, spread evenly (in their
                               logarithm) from `nodes` to `nodes_last`
  points, points_last          points per state, spread the same way
  cloud  "uniform" in the unit cube, or "mixed": half uniform, half N(0.5, 0.05^2)
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "hddm-solver-postprocessors_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import hddm_b200 as H  # noqa: E402

MAX_LEVEL = 7


def _case(call, form, dim, total_dof, nodes, points, states=1, nodes_last=None, points_last=None, level=0,
          cloud="uniform", want_surplus=True):
    return {"call": call, "form": form, "dim": dim, "total_dof": total_dof, "states": states, "level": level,
            "nodes": nodes, "nodes_last": nodes_last or nodes, "points": points, "points_last": points_last or points,
            "cloud": cloud, "want_surplus": want_surplus}


def listed():
    cases = {
        # the solver's own call: one point, host arrays in and out
        "host_one_point": _case("host", "fp64", 59, 118, 100_000, 1),
        # the solver's multistate call: one point in each of 16 states
        "host_16_states": _case("host", "fp64", 59, 118, 16_000, 1, states=16, nodes_last=30_000),
        # a handful of points of one state, such as one rank's share of a small step
        "few_points_fp32c": _case("device", "fp32c", 59, 118, 60_000, 75),
        # a rank's points of one solver step
        "step_fp64": _case("device", "fp64", 59, 118, 150_000, 1_500, cloud="mixed"),
        # the same on wide rows in the compensated form
        "step_fp32c": _case("device", "fp32c", 59, 256, 70_000, 10_007, cloud="mixed"),
        # a regular grid (shallow, wide tree), where every point has thousands of active nodes
        "regular_fp64": _case("device", "fp64", 16, 32, 51_137, 65_536, level=5),
        # a multistate set with ragged batches in one call, both forms
        "set_fp64": _case("device", "fp64", 30, 64, 20_000, 1_003, states=6, nodes_last=150_000, points_last=100_000),
        "set_fp32c": _case("device", "fp32c", 30, 64, 20_000, 1_003, states=6, nodes_last=150_000, points_last=100_000),
        # throughput: grids whose rows exceed the L2, batches above the chunking threshold
        "large_fp64": _case("device", "fp64", 59, 256, 150_000, 131_072, cloud="mixed"),
        "large_fp32c": _case("device", "fp32c", 59, 256, 140_000, 262_144, cloud="mixed"),
        # training: gradients for the points and for every surplus
        "grad_batch": _case("grad", "fp64", 59, 128, 300_000, 32_768),
        # sensitivities: gradients for the points alone, an odd batch
        "grad_x": _case("grad", "fp64", 59, 118, 50_000, 5_001, want_surplus=False),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("host", "few", "step", "set", "large", "regular", "grad"))
    form = rng.choice(("fp64", "fp32c"))
    dim = rng.choice((10, 16, 30, 45, 59, 59))
    td = rng.choice((8, 32, 37, 64, 118, 118, 128, 200, 256))
    cloud = rng.choice(("uniform", "mixed"))
    rows = 30_000_000 // td                      # nodes of all states together
    if kind == "host":
        states = rng.choice((1, 1, 4, 16))
        n = _log(rng, 10_000, min(200_000, rows // states))
        return _case("host", "fp64", dim, td, n, rng.choice((1, 1, 2, 3)), states=states,
                     nodes_last=max(10_000, n * 2 // 3), cloud=cloud)
    if kind == "few":
        return _case("device", form, dim, td, _log(rng, 10_000, min(200_000, rows)), _log(rng, 4, 1_100), cloud=cloud)
    if kind == "step":
        return _case("device", form, dim, td, _log(rng, 10_000, min(200_000, rows)), _log(rng, 1_100, 30_000), cloud=cloud)
    if kind == "set":
        states = rng.choice((3, 6, 8))
        n, last = (_log(rng, 10_000, max(11_000, min(150_000, rows // states))) for _ in range(2))
        p, q = (_log(rng, 100, 60_000) for _ in range(2))
        return _case("device", form, dim, td, n, p, states=states, nodes_last=last, points_last=q, cloud=cloud)
    if kind == "large":
        n = _log(rng, 30_000, min(200_000, rows))
        return _case("device", form, dim, td, n, _log(rng, 60_000, min(200_000, 25_000_000 // td)), cloud=cloud)
    if kind == "regular":
        dim, level = rng.choice(((4, 4), (10, 4), (16, 4), (10, 5), (16, 5)))
        td = rng.choice((8, 32, 37, 64))
        return _case("device", form, dim, td, 0, _log(rng, 1_000, 30_000), level=level)
    td = rng.choice((8, 32, 64, 118, 128))
    return _case("grad", "fp64", dim, td, _log(rng, 10_000, min(200_000, rows)), _log(rng, 200, 20_000), cloud=cloud,
                 want_surplus=rng.random() < 0.6)


# ------------------------------------------------------------------- inputs
def _spread(first, last, n):
    if n == 1:
        return [first]
    return [int(round(first * (last / first) ** (k / (n - 1)))) for k in range(n)]


def _host_grids(case, seed):
    sizes = _spread(max(case["nodes"], 1), max(case["nodes_last"], 1), case["states"])
    if case["level"]:
        return [H.HostGrid.regular(case["dim"], case["level"], case["total_dof"], seed=seed + k)
                for k in range(case["states"])]
    return [H.HostGrid.adaptive(case["dim"], n, case["total_dof"], seed=16 * seed + k, max_level=MAX_LEVEL)
            for k, n in enumerate(sizes)]


def _counts(case):
    # the state with the most nodes does not have the most points
    c = _spread(case["points"], case["points_last"], case["states"])
    return c[1::2] + c[0::2]


def _points(case, seed):
    """Device points (states in order), and for "grad" dL/dvalue."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, dim = sum(_counts(case)), case["dim"]
    x = torch.rand((n, dim), generator=gen, dtype=torch.float64, device="cuda")
    if case["cloud"] == "mixed":
        h = n // 2
        x[h:] = (0.5 + 0.05 * torch.randn((n - h, dim), generator=gen, dtype=torch.float64, device="cuda")).clamp_(0, 1)
    gout = None
    if case["call"] == "grad":
        gout = torch.randn((n, case["total_dof"]), generator=gen, dtype=torch.float64, device="cuda")
    return x, gout


def prepare(case, seed):
    flags = H.BUILD_FP32 if case["form"] == "fp32c" else 0
    grids = [H.Grid(h, flags=flags) for h in _host_grids(case, seed)]
    x, gout = _points(case, seed)
    if case["call"] == "host":
        x = x.cpu().numpy()
    return {"case": case, "grids": grids, "counts": _counts(case), "x": x, "gout": gout,
            "precision": H.FP32C if case["form"] == "fp32c" else H.FP64}


def run(state):
    call = state["case"]["call"]
    if call == "host":
        return H.interpolate_host(state["grids"], state["x"], counts=state["counts"], precision=state["precision"])
    if call == "device":
        return H.interpolate(state["grids"], state["x"], counts=state["counts"], precision=state["precision"])
    gx, gs = H.backward(state["grids"][0], state["x"], state["gout"], want_surplus=state["case"]["want_surplus"])
    return {"x": gx, "surplus": gs} if gs is not None else {"x": gx}


# --------------------------------------------------------------------- work
def _active(case, nodes):
    """Active nodes per point, as counted on grids of these kinds (the mean
    over grids and points; single grids differ by a factor of about two)."""
    if case["level"]:
        return float(math.comb(case["dim"] + case["level"] - 1, case["level"] - 1))
    return min(nodes, min(7.0 * case["dim"], 300.0) * math.sqrt(nodes / 20_000))


def work(case):
    dim, td, nbytes, flops = case["dim"], case["total_dof"], 0.0, 0.0
    sizes = _spread(max(case["nodes"], 1), max(case["nodes_last"], 1), case["states"])
    for nodes, npts in zip(sizes, _counts(case)):
        if case["level"]:
            nodes = _regular_nodes(dim, case["level"])
        pairs = npts * _active(case, nodes)
        row = td * (8 if case["form"] == "fp64" else 4)
        nbytes += npts * (dim + td) * 8 + min(nodes, pairs) * row
        flops += 2 * td * pairs
        if case["call"] == "grad":
            nbytes += npts * dim * 8
            if case["want_surplus"]:
                nbytes += nodes * td * 8
                flops += 2 * td * pairs
    return {"bytes": nbytes, "flops": flops}


def _regular_nodes(dim, level):
    """Nodes of a regular grid: 1, 2, 2, 4, 8, ... of them per dimension at level 1, 2, 3, ..."""
    per = [1, 2] + [1 << (l - 2) for l in range(3, level + 1)]
    ways = [1] + [0] * (level - 1)
    for _ in range(dim):
        ways = [sum(ways[s - l] * per[l] for l in range(s + 1)) for s in range(level)]
    return sum(ways)


# -------------------------------------------------------------------- exact
DENSE = 4            # hats evaluated for every (point, node) before the pairs are listed
BLOCK = 1 << 25      # (point, node) products per block


def _hat(x, i, j):
    return 1.0 - (x * i - j).abs()


class _Grid64:
    """A host grid's arrays as device tensors: the non-constant (dim, i, j) of
    every node, padded with i = j = 0 (a hat of 1), and the surplus rows."""

    def __init__(self, host):
        index, surplus = host.arrays()
        dim = index.shape[1] // 2
        used = (index[:, :dim] != 0) | (index[:, dim:] != 0)
        width = max(1, int(used.sum(1).max()))
        order = np.argsort(~used, axis=1, kind="stable")[:, :width]
        keep = np.take_along_axis(used, order, 1)
        i = np.where(keep, np.take_along_axis(index[:, :dim], order, 1), 0)
        j = np.where(keep, np.take_along_axis(index[:, dim:], order, 1), 0)
        dev = dict(device="cuda")
        self.dims = torch.as_tensor(order, **dev)
        self.i, self.j = torch.as_tensor(i, dtype=torch.float64, **dev), torch.as_tensor(j, dtype=torch.float64, **dev)
        self.surplus = torch.as_tensor(surplus, **dev)
        self.width, self.n = width, len(index)

    def pairs(self, x):
        """(point, node) index tensors of every pair whose hats are all positive, block by block."""
        step = max(1, BLOCK // self.n)
        for b in range(0, len(x), step):
            xb = x[b:b + step]
            alive = torch.ones((len(xb), self.n), dtype=torch.bool, device="cuda")
            for c in range(min(DENSE, self.width)):
                alive &= _hat(xb[:, self.dims[:, c]], self.i[:, c], self.j[:, c]) > 0
            p, n = alive.nonzero(as_tuple=True)
            for c in range(DENSE, self.width):
                ok = _hat(xb[p, self.dims[n, c]], self.i[n, c], self.j[n, c]) > 0
                p, n = p[ok], n[ok]
            for q in range(0, len(p), 1 << 19):
                yield p[q:q + (1 << 19)] + b, n[q:q + (1 << 19)]

    def hats(self, x, p, n):
        return _hat(x[p[:, None], self.dims[n]], self.i[n], self.j[n])


def exact(case, seed):
    hosts = _host_grids(case, seed)
    x, gout = _points(case, seed)
    if case["call"] == "grad":
        g = _Grid64(hosts[0])
        gx, gs = torch.zeros_like(x), torch.zeros_like(g.surplus)
        for p, n in g.pairs(x):
            h = g.hats(x, p, n)
            ones = torch.ones_like(h[:, :1])
            before = torch.cumprod(torch.cat([ones, h[:, :-1]], 1), 1)
            after = torch.cumprod(torch.cat([ones, h.flip(1)[:, :-1]], 1), 1).flip(1)
            slope = -g.i[n] * torch.sign(x[p[:, None], g.dims[n]] * g.i[n] - g.j[n])
            cs = (gout[p] * g.surplus[n]).sum(1, keepdim=True)
            gx.view(-1).index_add_(0, (p[:, None] * x.shape[1] + g.dims[n]).view(-1), (cs * before * after * slope).view(-1))
            if case["want_surplus"]:
                gs.index_add_(0, n, h.prod(1, keepdim=True) * gout[p])
        return {"x": gx, "surplus": gs} if case["want_surplus"] else {"x": gx}
    out = torch.zeros((len(x), case["total_dof"]), dtype=torch.float64, device="cuda")
    at = 0
    for host, count in zip(hosts, _counts(case)):
        g, xs = _Grid64(host), x[at:at + count]
        for p, n in g.pairs(xs):
            out.index_add_(0, p + at, g.hats(xs, p, n).prod(1, keepdim=True) * g.surplus[n])
        at += count
    return out.cpu().numpy() if case["call"] == "host" else out
