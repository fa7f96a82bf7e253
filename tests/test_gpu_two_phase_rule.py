"""Up to how many points a batch takes the two-phase kernels: on either side of
each line, the way taken (from the launch statistics) and the results; and on
shapes where two phases took about twice as long as the one-phase kernels, that
a call is no slower than those (sgi_interpolate_noalloc runs them)."""
import ctypes

import numpy as np
import pytest

import hddm_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu
REGULAR, SPARSE = ("regular", 16, 4), ("adaptive", 10, 60_000)   # a point meets a sixth, and 1/680, of the nodes


def _host(kind, td):
    return (H.HostGrid.regular(kind[1], kind[2], td, seed=3) if kind[0] == "regular"
            else H.HostGrid.adaptive(kind[1], kind[2], td, seed=80))


def _warps():
    import torch
    return 8 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("kind,td,precision,npts,two", [
    (REGULAR, 37, H.FP64, -1, True), (REGULAR, 37, H.FP64, 0, False), (REGULAR, 64, H.FP64, 1500, False),
    (("regular", 10, 5), 130, H.FP64, 250, True), (("regular", 10, 5), 130, H.FP64, 350, False), (("regular", 16, 5), 130, H.FP64, 300, True),
    (REGULAR, 118, H.FP32C, -1, True), (REGULAR, 118, H.FP32C, 0, False),
    (SPARSE, 33, H.FP32C, -1, False), (SPARSE, 33, H.FP32C, 300 - 8 * 148, True),
    (("adaptive", 59, 150_000), 118, H.FP32C, 120 - 8 * 148, True),
    (("adaptive", 59, 150_000), 118, H.FP32C, 700 - 8 * 148, False),
    (("adaptive", 59, 150_000), 118, H.FP64, 300, True)])
def test_either_side_of_the_line(cuda, kind, td, precision, npts, two):
    """npts: beyond the number of warps that the GPU holds (counts below it are
    given for 148 SMs)."""
    import torch
    n = _warps() + npts
    hg = _host(kind, td)
    X = H.gen_points(kind[1], n, kind=0, seed=1)
    g = H.Grid(hg, flags=H.BUILD_FP32)
    out = H.interpolate(g, torch.from_numpy(X).cuda(), precision=precision).cpu().numpy()
    assert (H.last_launch().kernels == 2) == two
    ref = O.Gold(*hg.arrays()).interpolate(X[::7], nthreads=4)
    if precision == H.FP64:
        assert np.array_equal(out[::7], ref)
    else:
        assert O.rel_error(out[::7], ref)[0] <= 1e-7


@pytest.mark.parametrize("kind,td,precision,npts", [
    (REGULAR, 64, H.FP64, 2700), (REGULAR, 8, H.FP64, 3700), (("regular", 10, 5), 118, H.FP64, 2000),
    (SPARSE, 64, H.FP32C, 1100), (SPARSE, 200, H.FP32C, 1000)])
def test_no_slower_than_one_phase(cuda, kind, td, precision, npts):
    import torch
    g = H.Grid(_host(kind, td), flags=H.BUILD_FP32)
    x = torch.from_numpy(H.gen_points(kind[1], npts, kind=0, seed=1)).cuda()
    out = torch.empty((npts, td), dtype=torch.float64, device="cuda")
    offs = np.array([0, npts], np.int64)
    f = H.lib.sgi_interpolate_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                  ctypes.c_void_p]
    arr = (ctypes.c_void_p * 1)(g.handle.value)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def one_phase():
        assert f(1, arr, offs.ctypes.data, x.data_ptr(), out.data_ptr(), precision, stream) == 0

    def default():
        H.interpolate(g, x, precision=precision)

    def best(call):
        times = []
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(10):
                call()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[1:])

    t1, t = best(one_phase), best(default)
    assert t <= 1.3 * t1, (t1, t)
