"""Plans share a tuned chunk size and variant by call shape; grids of equal
sizes whose points meet many or few nodes take other kernels, and are tuned
apart."""
import pytest

import hddm_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,dim,td", [(H.FP64, 16, 256), (H.FP32C, 10, 32)])
def test_grids_that_take_other_kernels_are_tuned_apart(cuda, precision, dim, td):
    import torch
    x = torch.rand((1500, dim), dtype=torch.float64, device="cuda")
    out = torch.empty((1500, td), dtype=torch.float64, device="cuda")

    def tuned(host):
        plan = H.Plan(H.Grid(host, flags=H.BUILD_FP32), x, out, precision=precision)
        return plan.tuned_ms

    idx, sur = H.HostGrid.regular(dim, 5, td, seed=1).arrays()     # 4,845 and 1,001 active nodes a point
    even = tuned(H.HostGrid.from_dense(idx, sur))
    few = [tuned(H.HostGrid.adaptive(dim, len(idx), td, seed=s)) for s in (2, 3)]    # a few hundred, tens
    assert few[0] == few[1] > 0.0          # one shape, tuned once
    assert even != few[0] and even > 0.0
