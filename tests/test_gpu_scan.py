"""Prefix sums of interval lengths and the curves' lengths they write: interval
counts at the edges of tiles (1,024 intervals, 8,192 from 786,433 intervals on),
curves that span several tiles, runs of curves within one tile, and curves without
intervals (a single control point) before, between and after others.

The curves are polylines (degree 1, integer edges of a 3-4-5 triangle), so every
interval's length is 5 and every prefix sum a whole number below 2^53: the result
is exact up to the rounding of each interval's own length, in float-float at most
28 units of 2^-46 (4e-13).
"""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu


def polylines(n_edges):
    n_edges = np.asarray(n_edges, np.int64)
    n = n_edges.size
    steps = np.tile([[3.0, 4.0], [4.0, -3.0]], (int(n_edges.max()) // 2 + 1, 1))
    path = np.r_[[[0.0, 0.0]], np.cumsum(steps, 0)]
    knots = [np.r_[0.0, np.arange(m + 1.0), float(m)] for m in n_edges]
    ctrl = [path[: m + 1].ravel() for m in n_edges]
    return ds._pack(np.ones(n), np.ones(n), np.full(n, 2), n_edges + 3, np.concatenate(knots), 2 * (n_edges + 1),
                    np.concatenate(ctrl), np.full(n, 3), "polylines", 1e-9)


CASES = {
    "one interval": [1],
    "a tile": [1024],
    "a tile and one": [1025],
    "one short of a tile": [1023],
    "tiles of single intervals": [1] * 2049,
    "curves over several tiles": [5000, 1, 1, 3000, 7],
    "heads at every place": list(range(1, 70)),
    "most for short tiles": [3 << 18],
    "one more": [(3 << 18) - 5, 3, 3],
    "without intervals": [0, 0, 3, 0, 2000, 0, 0, 0, 1, 0],
    "none with intervals": [0, 0, 0],
    "long tiles": [8192 * 3, 8191, 1, 1] + [777] * 1400,
}


@pytest.mark.parametrize("precision", [g.GCV_PLAIN_FP64, g.GCV_MIXED])
@pytest.mark.parametrize("name", CASES)
def test_curve_lengths_and_sums(name, precision, gpu_lib):
    m = np.array(CASES[name])
    b = polylines(m)
    with g.ArclengthCalculateGpu.from_batch(b, precision=precision, rtol=1e-9) as calc:
        for _ in range(2):
            calc.createArclengthTable()
            np.testing.assert_allclose(calc.getAllCurveArclengths(), 5.0 * m, rtol=4e-13)
        # the sums inside the curves: the middle of the length is the middle of the parameter
        u = calc.arclengthReverse(b.n_samples, np.tile([0.25, 0.5, 1.0], m.size), True, g.GCV_HOST).us.reshape(-1, 3)
        np.testing.assert_allclose(u, m[:, None] * np.array([0.25, 0.5, 1.0]), rtol=1e-8)
