"""FP64 curves with infinite or NaN control values: the lengths and samples of the walk
with a float-float partition are those of the FP64 walk (below rtol 1e-12), curve by
curve, and the other curves are as without them."""
import ctypes

import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu

BAD = [np.inf, -np.inf, np.nan]


def curves(p, d, bad):
    """Twelve B-splines; every second one has a control value replaced, at another place each time."""
    rng = np.random.default_rng(10 * p + d)
    nc = np.full(12, p + 6)
    nk, knots, clen, ctrl = ds._random_knot_bsplines(rng, np.full(12, p), np.full(12, d), nc, 1.0)
    b = ds._pack(np.ones(12), np.full(12, p), np.full(12, d), nk, knots, clen, ctrl, np.full(12, 9), "bad", 1e-10)
    for i in range(0, 12, 2):
        b.ctrl[b.ctrl_off[i] + (i * (p + 5) * d // 10)] = bad
    return b


def run(b, rtol, relative):
    calc = g.ArclengthCalculateGpu.from_batch(b, precision=g.GCV_PLAIN_FP64, rtol=rtol, max_depth=20)
    calc.createArclengthTable()
    pos = np.tile(np.linspace(0.0, 1.0, 9), b.n_curve)
    return calc.getAllCurveArclengths(), calc.arclengthReverse(b.n_samples, pos, relative, g.GCV_HOST).us


@pytest.mark.parametrize("relative", [True, False])
@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("p,d", [(1, 2), (2, 3), (3, 2), (5, 3)])
def test_curves(p, d, bad, relative, gpu_lib):
    b = curves(p, d, bad)
    (L, u), (want_L, want_u) = run(b, 1e-10, relative), run(b, 0.5e-12, relative)
    np.testing.assert_allclose(L, want_L, rtol=1e-9)
    # (the FP64 Newton has no threshold to stop at where the length is NaN)
    np.testing.assert_allclose(u, want_u, atol=1e-8 if relative else 1e-5)


@pytest.mark.parametrize("bad", BAD)
def test_lengths_without_a_table(bad, gpu_lib):
    torch = pytest.importorskip("torch")
    b = curves(3, 2, bad)
    ko = torch.from_numpy(b.knot_off.astype(np.int32)).cuda()
    kv, cp = torch.from_numpy(b.knots).cuda(), torch.from_numpy(b.ctrl).cuda()
    q = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    out = []
    for rtol in (1e-10, 0.5e-12):
        x = torch.empty(b.n_curve, dtype=torch.float64, device="cuda")
        assert gpu_lib.gcv_bspline_lengths_noalloc(b.n_curve, 3, 2, q(ko), q(kv), q(cp), rtol, 20, q(x), None, None) == 0
        out.append(x.cpu().numpy())
    np.testing.assert_allclose(out[0], out[1], rtol=1e-9)
