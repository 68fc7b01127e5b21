"""A captured step whose pools turn out too small for the data: the control points
behind a captured step become curves with far more leaves than the pool and the deep
list were sized for.  The sampler of that replay reads no table entry, the step is run
again, and its results are those of a new context, bit for bit."""
import numpy as np
import pytest

import gcurval_gb300 as g
from test_gpu_walk import Cusps

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def device(b):
    tk = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dt)  # noqa: E731
    return ((tk(b.kind, torch.uint8), tk(b.degree, torch.uint8), tk(b.dim, torch.uint8), tk(b.knot_off, torch.int64),
             tk(b.knots, torch.float64), tk(b.ctrl_off, torch.int64), tk(b.ctrl, torch.float64)),
            tk(b.n_samples, torch.int32), tk(b.sample_positions(), torch.float64))


@pytest.mark.parametrize("what", [g.GCV_RETURN_US, g.GCV_RETURN_POINTS])
@pytest.mark.parametrize("kw", [dict(precision=g.GCV_PLAIN_FP64, rtol=1e-12), dict(precision=g.GCV_PLAIN_FP64, rtol=5e-13),
                                dict(precision=g.GCV_MIXED, rtol=1e-11),
                                dict(precision=g.GCV_MIXED, rtol=1e-11, mapping="half_warp")],
                         ids=["fp64", "fp64_tight", "mixed", "mixed_half_warp"])
def test_replay_that_outgrows_the_pools(kw, what, gpu_lib):
    n = 6000
    many = Cusps(500, 4, seed=41).batch
    many = many.subset(np.arange(n) % 500)
    arrays, counts, pos = device(many)
    width = 1 if what == g.GCV_RETURN_US else 2
    out, want = (torch.empty(pos.shape[0] * width, dtype=torch.float64, device="cuda") for _ in range(2))
    ref = g.ArclengthCalculateGpu.from_device_batch(*arrays, **kw)
    ref.createArclengthTable()
    ref.arclengthReverseInto(counts, pos, want, True, what)
    ctrl = arrays[6]
    bent = ctrl.clone()
    # straight and evenly parametrised: one leaf an interval
    ctrl.view(n, 6, 2).copy_(torch.arange(6, dtype=torch.float64, device="cuda")[None, :, None].expand(n, 6, 2))
    calc = g.ArclengthCalculateGpu.from_device_batch(*arrays, **kw)
    calc.stepGraph(counts, pos, out, True, what)
    calc.stepGraph(counts, pos, out, True, what)
    assert calc.stats()["n_leaves"] == n
    ctrl.copy_(bent)
    for _ in range(3):  # the replay that overflows, the next capture, its replay
        out.fill_(-7.0)
        calc.stepGraph(counts, pos, out, True, what)
        np.testing.assert_array_equal(calc.getAllCurveArclengths(), ref.getAllCurveArclengths())
        np.testing.assert_array_equal(out.cpu().numpy(), want.cpu().numpy())
    assert calc.stats()["n_leaves"] > 3 * n + 4096
