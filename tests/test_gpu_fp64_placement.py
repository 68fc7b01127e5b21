"""Samples of FP64 tables stop within a tenth of rtol of the curve's length, also at
tolerances where the float-float Newton step's own FP32 rounding is not far below that.

Bound: a tenth of rtol, a tenth of that for the residual being an estimate, and 1e-12
for the oracle's lengths, the table's own error being far below at these tolerances.
"""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds
from oracle.oracle import ScaledOracle

pytestmark = pytest.mark.gpu


def curves(seed, n_samples=201):
    """300 B-splines of every degree and dimension, 0 to 11 random inner knots."""
    rng = np.random.default_rng(seed)
    deg, dim = rng.integers(1, 6, 300), rng.integers(2, 4, 300)
    nc = deg + 1 + rng.integers(0, 12, 300)
    nk, knots, clen, ctrl = ds._random_knot_bsplines(rng, deg, dim, nc, 1.0)
    return ds._pack(np.ones(300), deg, dim, nk, knots, clen, ctrl, np.full(300, n_samples), "p", 1e-9)


@pytest.fixture(scope="module")
def batch():
    b = curves(5)
    pos = np.random.default_rng(6).random(b.total_samples)
    o = ScaledOracle(b)
    return b, pos, o, o.lengths()


@pytest.mark.parametrize("rtol", [1e-8, 3e-9, 1e-9, 5e-10, 1e-10])
def test_samples_within_a_tenth(rtol, batch, gpu_lib):
    b, pos, oracle, lengths = batch
    calc = g.ArclengthCalculateGpu.from_batch(b, precision=g.GCV_PLAIN_FP64, rtol=rtol)
    calc.createArclengthTable()
    table = np.abs(calc.getAllCurveArclengths() - lengths) / lengths
    u = calc.arclengthReverse(b.n_samples, pos, True, g.GCV_HOST).us
    L = np.repeat(lengths, b.n_samples)
    err = np.abs(oracle.s_at(b.n_samples, u) - pos * L) / L
    smooth = np.repeat(table < 0.01 * rtol, b.n_samples)  # (a near-cusp accepted by accident moves the length)
    assert smooth.mean() > 0.9
    assert err[smooth].max() <= 0.11 * rtol + 1e-12
