"""FP64 lengths of pieces whose speed has a zero of even order, inside or at an end:
the speed is a polynomial there, so the first panels are accepted and the length is as
good as the speeds at their nodes, also at the nodes next to the zero.

C' = (t - r)^m e with a fixed vector e: the length is |e| ((1 - r)^(m+1) + r^(m+1)) / (m + 1).
Tolerance: the Kronrod rule is exact for these speeds, and set-up, speeds and the sum
of fifteen terms carry some twenty roundings of 2^-53 of the largest speed, which is
at most (m + 1) 2^m times the mean: 64 * 2^-53 * 16 * 5 is the bound at m = 4.
"""
import ctypes
from math import comb

import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds
from gcurval_gb300 import learned

pytestmark = pytest.mark.gpu

CASES = [(p, d, m) for p in (3, 4, 5) for d in (2, 3) for m in (2, 4) if m < p]


def depth_network(depth):
    """Weights of a network that predicts `depth` with equal quarters for every interval."""
    w = np.zeros(learned.N_PARAM, np.float32)
    w[-32 + depth] = 8.0  # the output layer's biases come last, the depth classes first
    return w


def pieces(p, d, m):
    """Bezier pieces of degree p with the zero at 0, at 1, at panel midpoints and between; their lengths."""
    rng = np.random.default_rng(100 * p + 10 * d + m)
    r = np.r_[0.0, 1.0, 0.5, 0.25, 0.5 + 0.5 * np.array([0.2077849550078985, -0.5860872354676911]), rng.random(60)]
    bern = np.array([[comb(j, i) / comb(p, i) if j >= i else 0.0 for i in range(p + 1)] for j in range(p + 1)])
    ctrl, want = [], []
    for ri in r:
        e = rng.normal(size=d)
        a = np.polyint(np.poly1d([ri] * m, r=True)).c[::-1]
        c = np.zeros(p + 1)
        c[:a.size] = a
        ctrl.append(((bern @ c)[:, None] * e).reshape(-1))
        want.append(np.linalg.norm(e) * ((1 - ri) ** (m + 1) + ri ** (m + 1)) / (m + 1))
    n = r.size
    b = ds._pack(np.ones(n), np.full(n, p), np.full(n, d), np.full(n, 2 * p + 2), np.tile(np.repeat([0.0, 1.0], p + 1), n),
                 np.full(n, (p + 1) * d), np.concatenate(ctrl), np.full(n, 9), "zeros", 1e-12)
    return b, np.array(want)


@pytest.mark.parametrize("learned_depth", [None, 3, 8])
@pytest.mark.parametrize("rtol", [1e-9, 1e-12])
@pytest.mark.parametrize("p,d,m", CASES)
def test_lengths(p, d, m, rtol, learned_depth, gpu_lib):
    b, want = pieces(p, d, m)
    calc = g.ArclengthCalculateGpu.from_batch(b, precision=g.GCV_PLAIN_FP64, rtol=rtol, learned=learned_depth is not None)
    if learned_depth is not None:
        calc.set_learned_model(depth_network(learned_depth))
    calc.createArclengthTable()
    np.testing.assert_allclose(calc.getAllCurveArclengths(), want, rtol=64 * 2.0 ** -53 * (m + 1) * 2 ** m)


@pytest.mark.parametrize("p,d,m", CASES)
def test_lengths_without_a_table(p, d, m, gpu_lib):
    torch = pytest.importorskip("torch")
    b, want = pieces(p, d, m)
    ko = torch.from_numpy(b.knot_off.astype(np.int32)).cuda()
    kv, cp = torch.from_numpy(b.knots).cuda(), torch.from_numpy(b.ctrl).cuda()
    out = torch.empty(b.n_curve, dtype=torch.float64, device="cuda")
    q = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert gpu_lib.gcv_bspline_lengths_noalloc(b.n_curve, p, d, q(ko), q(kv), q(cp), 1e-12, 30, q(out), None, None) == 0
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=64 * 2.0 ** -53 * (m + 1) * 2 ** m)
