"""Knots in any unit: a curve's length does not depend on the unit of its knots,
its parameters scale with it, its points stay, whatever the unit of its coordinates.

Knots and coordinates are scaled by powers of two, so every step of the set-up, the
walk and the sampler is the unscaled one but for bits lost below the smallest number of
the format: none in FP64 (2^-1000 times spans of 2^-5 and more), and in float-float
(2^-100, FP32's smallest 2^-149) at most 2^-44 of a span, 1e-12 with the few terms and
the condition of such curves.  A sample is within rtol of the length either way, and the curves
move by at least half their length per knot range.
"""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu


def curves(knot_power, coord_power, short=None):
    """One curve per degree and dimension; short: the first span's width before scaling."""
    rng = np.random.default_rng(31)
    deg, dim, nk, nc, knots, ctrl = [], [], [], [], [], []
    for p in range(1, 6):
        for d in (2, 3):
            inner = np.linspace(0.1, 0.9, 8) + 0.02 * rng.uniform(-1, 1, 8)
            if short:
                inner[0] = short
            k = np.r_[np.zeros(p + 1), inner, np.ones(p + 1)]
            n = k.size - p - 1
            c = np.c_[np.linspace(0, 1, n), 0.1 * rng.normal(size=(n, d - 1))].reshape(-1)
            deg.append(p), dim.append(d), nk.append(k.size), nc.append(c.size)
            knots.append(k * 2.0 ** knot_power), ctrl.append(c * 2.0 ** coord_power)
    return ds._pack(np.ones(len(deg)), deg, dim, nk, np.concatenate(knots), nc, np.concatenate(ctrl),
                    np.full(len(deg), 33), "units", 1e-10)


def run(b, precision, rtol):
    calc = g.ArclengthCalculateGpu.from_batch(b, precision=precision, rtol=rtol)
    calc.createArclengthTable()
    pos = b.sample_positions()
    return (calc.getAllCurveArclengths(), calc.arclengthReverse(b.n_samples, pos, True, g.GCV_HOST).us,
            calc.arclengthReverse(b.n_samples, pos, True, g.GCV_HOST, g.GCV_RETURN_POINTS).points)


@pytest.mark.parametrize("precision,rtol,knot_power,coord_power",
                         [(g.GCV_MIXED, 1e-9, k, c) for k in (-100, -30, 100) for c in (-30, 0, 30)] +
                         [(g.GCV_PLAIN_FP64, r, k, c) for r in (1e-10, 0.9e-12) for k in (-1000, -900, 1000)
                          for c in (-30, 0, 30)])
def test_units(precision, rtol, knot_power, coord_power, gpu_lib):
    L0, _, p0 = run(curves(0, 0), precision, rtol)
    L, _, p = run(curves(knot_power, coord_power), precision, rtol)
    np.testing.assert_allclose(L * 2.0 ** -coord_power, L0, rtol=1e-12)
    np.testing.assert_allclose(p * 2.0 ** -coord_power, p0, rtol=0, atol=20 * rtol)


@pytest.mark.parametrize("coord_power", [-30, 0, 30])
@pytest.mark.parametrize("precision,power", [(g.GCV_MIXED, -60), (g.GCV_MIXED, -100), (g.GCV_PLAIN_FP64, -100),
                                             (g.GCV_PLAIN_FP64, -900)])
def test_a_span_far_shorter_than_its_neighbours(precision, power, coord_power, gpu_lib):
    """The rest of the curve is as without it, and its own points are the curve's start."""
    L0, _, p0 = run(curves(0, 0, short=2.0 ** -40), precision, 1e-9)
    L, _, p = run(curves(0, coord_power, short=2.0 ** power), precision, 1e-9)
    np.testing.assert_allclose(L * 2.0 ** -coord_power, L0, rtol=1e-9)
    np.testing.assert_allclose(p * 2.0 ** -coord_power, p0, rtol=0, atol=1e-7)
