"""Curves without a knot interval (a single span's knots short) have length 0 wherever
they stand, in a table built over recycled memory too, and a long run of them takes no
longer than its memory: the prefix sums of two curves among 400,000 empty ones take less
than a tenth of a millisecond more than those of the two alone."""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu


def batch(empty_before, empty_between, empty_after):
    """Two cubics of 30 points with runs of empty cubics (7 knots, 3 points) around them."""
    rng = np.random.default_rng(9)
    two = ds.uniform_bsplines(2, n_ctrl=30, n_samples=3, seed=9)
    nk, nc, knots, ctrl, ns = [], [], [], [], []
    for i, run in enumerate((empty_before, empty_between, empty_after)):
        nk += [7] * run
        nc += [6] * run
        knots.append(np.tile(np.arange(7.0), run))
        ctrl.append(rng.normal(size=6 * run))
        if i < 2:
            nk.append(34)
            nc.append(60)
            knots.append(two.knots[34 * i:34 * (i + 1)])
            ctrl.append(two.ctrl[60 * i:60 * (i + 1)])
    n = len(nk)
    b = ds._pack(np.ones(n), np.full(n, 3), np.full(n, 2), nk, np.concatenate(knots), nc, np.concatenate(ctrl),
                 np.full(n, 1), "empties", 1e-9)
    return b, two, np.array([empty_before, empty_before + 1 + empty_between])


def build(b, precision, times=1):
    with g.ArclengthCalculateGpu.from_batch(b, precision=precision, rtol=1e-9, collect_stats=True) as calc:
        ms = []
        for _ in range(times):
            calc.createArclengthTable()
            ms.append(calc.stats()["ms_scan"])
        return calc.getAllCurveArclengths(), float(np.median(ms))


@pytest.mark.parametrize("precision", [g.GCV_PLAIN_FP64, g.GCV_MIXED])
@pytest.mark.parametrize("runs", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (5, 0, 3000), (3000, 2000, 0)])
def test_lengths(runs, precision, gpu_lib):
    b, two, at = batch(*runs)
    want, _ = build(two, precision)
    # a context of the same size whose lengths are not zero leaves its memory behind
    build(ds.uniform_bsplines(b.n_curve, n_ctrl=5, n_samples=1, seed=1), precision)
    L, _ = build(b, precision)
    np.testing.assert_array_equal(L[at], want)
    assert not np.delete(L, at).any()


def test_a_long_run_costs_a_clear(gpu_lib):
    b, two, _ = batch(0, 400_000, 0)
    _, alone = build(two, g.GCV_MIXED, times=15)
    _, among = build(b, g.GCV_MIXED, times=15)
    assert among <= alone + 0.1
