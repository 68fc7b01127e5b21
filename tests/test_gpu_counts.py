"""Device sample counts: checked and used in one reading by the library, with the
caller's stream waited for; what was refused stays refused with the same message."""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(params=["plain", "mixed", "f32", "several codes"])
def case(request, gpu_lib):
    if request.param == "several codes":
        b = ds.uneven_batch(40, seed=3, max_ctrl=60, max_samples=50)
    else:
        b = ds.uniform_bsplines(40, n_ctrl=12, n_samples=25, seed=4)
    prec = g.GCV_PLAIN_FP64 if request.param == "plain" else g.GCV_MIXED
    if request.param == "f32":
        ko = b.knot_off.astype(np.int32)
        calc = g.ArclengthCalculateGpu.bsplines(3, 2, ko, b.knots.astype(np.float32), b.ctrl.astype(np.float32),
                                                precision=prec, rtol=1e-6)
    else:
        calc = g.ArclengthCalculateGpu.from_batch(b, precision=prec, rtol=1e-8)
    calc.createArclengthTable()
    dt = torch.float32 if request.param == "f32" else torch.float64
    yield calc, b, dt
    calc.close()


def test_device_counts_equal_host_counts(case):
    calc, b, dt = case
    pos = torch.from_numpy(b.sample_positions()).to(dt)
    want = calc.arclengthReverse(b.n_samples, pos.numpy(), True, g.GCV_HOST).us
    # counts and positions still being written on a side stream when the call starts
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        n = torch.from_numpy(b.n_samples).cuda(non_blocking=True) * 1
        p = pos.cuda(non_blocking=True) * 1
        out = torch.full((b.total_samples,), -1.0, dtype=dt, device="cuda")
        calc.arclengthReverseInto(n.to(torch.int32), p, out)
        calc.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), want)


def test_refusals(case):
    calc, b, dt = case
    n = torch.from_numpy(b.n_samples).cuda()
    p = torch.from_numpy(b.sample_positions()).to(dt).cuda()
    out = torch.full((b.total_samples,), -1.0, dtype=dt, device="cuda")
    torch.cuda.synchronize()
    total = b.total_samples
    m = n.clone()
    m[3] += 1
    with pytest.raises(ValueError, match=f"add up to {total + 1}, {total} positions given"):
        calc.arclengthReverseInto(m, p, out)
    with pytest.raises(ValueError, match=f"add up to {total + 1}, {total} positions given"):
        calc.arclengthReverseInto(m, p, out[:-1])
    with pytest.raises(ValueError, match=f"output holds {total - 1} values, {total} needed"):
        calc.arclengthReverseInto(n, p, out[:-1])
    with pytest.raises(ValueError, match=f"39 sample counts for {b.n_curve} curves"):
        calc.arclengthReverseInto(n[:39], p, out)
    m = n.clone()
    m[0] += m[1] + 1
    m[1] = -1
    with pytest.raises(g.GcvError, match="negative sample count"):
        calc.arclengthReverseInto(m, p, out)
    calc.synchronize()
    assert bool((out == -1.0).all())
