"""A captured step is captured again when an ordinary build has replaced a buffer it
addresses: the leaf pool (a tighter tolerance in between) or the coefficients (the
other precision in between).  Its results are then those of a new context."""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds
from test_gpu_graph_pools import device

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LOOSE = dict(precision=g.GCV_PLAIN_FP64, rtol=1e-4)
MIXED = dict(precision=g.GCV_MIXED, rtol=1e-6)


@pytest.mark.parametrize("first,between", [(LOOSE, dict(precision=g.GCV_PLAIN_FP64, rtol=1e-13)), (MIXED, LOOSE),
                                           (LOOSE, MIXED), (MIXED, dict(precision=g.GCV_MIXED, rtol=1e-12))])
def test_step_after_a_build_with_other_options(first, between, gpu_lib):
    b = ds.uniform_bsplines(500, n_ctrl=30, n_samples=20, seed=6)
    arrays, counts, pos = device(b)
    out, want = (torch.empty(pos.shape[0], dtype=torch.float64, device="cuda") for _ in range(2))
    ref = g.ArclengthCalculateGpu.from_device_batch(*arrays, **first)
    ref.createArclengthTable()
    ref.arclengthReverseInto(counts, pos, want, True, g.GCV_RETURN_US)
    calc = g.ArclengthCalculateGpu.from_device_batch(*arrays, **first)
    for _ in range(5):  # until the launch shapes are settled
        calc.stepGraph(counts, pos, out)
    for _ in range(2):
        calc.set_options(between["precision"], rtol=between["rtol"])
        calc.createArclengthTable()
        filler = torch.full((4 << 20,), float("nan"), device="cuda")  # what was freed belongs to someone else now
        calc.set_options(first["precision"], rtol=first["rtol"])
        out.fill_(-7.0)
        calc.stepGraph(counts, pos, out)
        np.testing.assert_array_equal(calc.getAllCurveArclengths(), ref.getAllCurveArclengths())
        np.testing.assert_array_equal(out.cpu().numpy(), want.cpu().numpy())
        assert bool(torch.isnan(filler).all())
        del filler
