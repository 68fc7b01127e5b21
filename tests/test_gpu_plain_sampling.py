"""Sampling of FP64 tables: the in-leaf Newton in float-float (tolerances from
1e-12 up) and in FP64 (below), and data far outside FP32's exponent range.

Tolerance: the table is good to rtol * L and a sample stops within a tenth of
that, so a position is within 1.1 rtol L of its target; the oracle's own
lengths are good to about 1e-14 relative, taken as 1e-13 here.
"""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds
from oracle.oracle import ScaledOracle

pytestmark = pytest.mark.gpu

ORACLE_EPS = 1e-13


def curves(p, d, n=12, seed=0, n_samples=41):
    """n random-knot B-splines of degree p in d dimensions, p + 1 to p + 12 points (p = 0: ellipses)."""
    if p == 0:
        return ds.ellipses(n, n_samples=n_samples, seed=seed)
    rng = np.random.default_rng(1000 * seed + 10 * p + d)
    nc = rng.integers(p + 1, p + 13, n)
    nk, knots, clen, ctrl = ds._random_knot_bsplines(rng, np.full(n, p), np.full(n, d), nc, 1.0)
    return ds._pack(np.ones(n), np.full(n, p), np.full(n, d), nk, knots, clen, ctrl, np.full(n, n_samples), "p", 1e-10)


def sample(batch, pos, rtol, **kw):
    calc = g.ArclengthCalculateGpu.from_batch(batch, precision=g.GCV_PLAIN_FP64, rtol=rtol, **kw)
    calc.createArclengthTable()
    return calc.arclengthReverse(batch.n_samples, pos, True, g.GCV_HOST).us


def positions(batch, seed):
    """Random fractions with both ends among them."""
    pos = np.random.default_rng(seed).random(batch.total_samples)
    off = np.concatenate([[0], np.cumsum(batch.n_samples)])
    pos[off[:-1]], pos[off[1:] - 1] = 0.0, 1.0
    return pos


def position_error(oracle, batch, u, pos):
    L = np.repeat(oracle.lengths(), batch.n_samples)
    return np.max(np.abs(oracle.s_at(batch.n_samples, u) - pos * L) / L)


CODES = [(0, 2)] + [(p, d) for d in (2, 3) for p in (1, 2, 3, 4, 5)]


@pytest.mark.parametrize("rtol", [1e-8, 1e-10, 1e-12, 0.99e-12, 1e-13])
@pytest.mark.parametrize("p,d", CODES)
def test_positions_hold_at_every_tolerance(p, d, rtol, gpu_lib):
    b = curves(p, d)
    pos = positions(b, 3)
    assert position_error(ScaledOracle(b), b, sample(b, pos, rtol), pos) <= 1.1 * rtol + ORACLE_EPS


@pytest.mark.parametrize("power", [-300, -140, -60, 60, 140, 300])
@pytest.mark.parametrize("p,d", [(0, 2), (3, 2), (5, 3)])
def test_scaled_curves_sample_alike(p, d, power, gpu_lib):
    """Control values times 2^power: the same curve in other units, far beyond FP32's range."""
    rtol = 1e-10
    b = curves(p, d, seed=1)
    pos = positions(b, 4)
    big = b.subset(np.arange(b.n_curve))
    scale = np.full(big.ctrl.size, 2.0 ** power)
    if p == 0:
        scale.reshape(-1, 5)[:, 2] = 1.0  # the rotation angle
    big.ctrl = big.ctrl * scale
    assert position_error(ScaledOracle(b), b, sample(big, pos, rtol), pos) <= 1.1 * rtol + ORACLE_EPS


def test_nonfinite_curve_gives_its_start_and_leaves_the_others(gpu_lib):
    b = curves(3, 2, seed=2)
    pos = positions(b, 5)
    good = sample(b, pos, 1e-10)
    b.ctrl[b.ctrl_off[4] + 2] = np.nan
    u = sample(b, pos, 1e-10)
    off = np.concatenate([[0], np.cumsum(b.n_samples)])
    at = slice(off[4], off[5])
    assert np.all(u[at] == b.knots[b.knot_off[4] + 3])
    keep = np.ones(u.size, bool)
    keep[at] = False
    np.testing.assert_array_equal(u[keep], good[keep])
