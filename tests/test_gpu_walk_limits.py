"""The length walk's limits on an interval's leaves (16 from a learned start, 96
otherwise) depend on the interval alone: an interval built by itself, where every
round takes only its own panels, has the same length and samples, bit for bit, as
among thousands, where other intervals' panels take part in its rounds.

Curves: quintics with cusps whose trees have about as many leaves as the limit.  The
learned start is a network without weights whose biases predict depth 3 (eight panels)
for every interval.
"""
import numpy as np
import pytest

import gcurval_gb300 as g
from test_gpu_smooth_zeros import depth_network
from test_gpu_walk import GK, Cusps

pytestmark = pytest.mark.gpu

START = 3


def learned_leaves(ref, i, rtol):
    """Leaves of curve i's walk from 2^START panels, tolerance rtol times its chord."""
    x, wk, wg = GK
    fx, fy = ref.derv[i]
    tol = rtol * np.hypot(*(np.polyval(np.polyint(p.c), 1.0) for p in (fx, fy)))
    todo, leaves = [(k, START) for k in range(2 ** START)], 0
    while todo:
        k, depth = todo.pop()
        hw = 2.0 ** -depth
        v = -1.0 + (2 * k + 1) * hw + hw * x
        f = 0.5 * np.hypot(fx(0.5 * (v + 1)), fy(0.5 * (v + 1)))
        K, G = hw * (wk @ f), hw * (wg @ f)
        if abs(K - G) <= max(tol * hw, 50 * 2.0 ** -46 * abs(K)) or depth >= 44:
            leaves += 1
        else:
            todo += [(2 * k + 1, depth + 1), (2 * k, depth + 1)]
    return leaves


def table(b, network=None, **kw):
    calc = g.ArclengthCalculateGpu.from_batch(b, collect_stats=True, learned=network is not None, **kw)
    if network is not None:
        calc.set_learned_model(network)
    calc.createArclengthTable()
    L = calc.getAllCurveArclengths()
    u = calc.arclengthReverse(b.n_samples, b.sample_positions(), True, g.GCV_HOST).us.reshape(b.n_curve, -1)
    st = calc.stats()
    calc.close()
    return L, u, st


def same_alone_as_among_others(b, pick, network=None, **kw):
    """Copies of every curve in random order, enough for thirty intervals per warp and more."""
    copies = -(-150_000 // b.n_curve)
    order = np.random.default_rng(7).permutation(np.repeat(np.arange(b.n_curve), copies))
    L, u, _ = table(b.subset(order), network, **kw)
    first = np.zeros(b.n_curve, np.int64)
    first[order[::-1]] = np.arange(order.size)[::-1]
    np.testing.assert_array_equal(L, L[first[order]])
    np.testing.assert_array_equal(u, u[first[order]])
    for i in pick:
        L1, u1, _ = table(b.subset(np.array([i])), network, **kw)
        np.testing.assert_array_equal(L1[0], L[first[i]], err_msg=f"curve {i}")
        np.testing.assert_array_equal(u1[0], u[first[i]], err_msg=f"curve {i}")


def few_samples(ref):
    ref.batch.n_samples[:] = 5
    return ref.batch


@pytest.mark.parametrize("precision", [g.GCV_MIXED, g.GCV_PLAIN_FP64])
@pytest.mark.parametrize("rtol", [1e-5, 1e-6])
def test_learned_starts_near_the_limit(rtol, precision, gpu_lib):
    ref = Cusps(400, 3, seed=21)
    leaves = np.array([learned_leaves(ref, i, rtol) for i in range(400)])
    pick = np.flatnonzero((leaves >= 15) & (leaves <= 30))
    assert np.sum((leaves > 16) & (leaves <= 30)) >= 80
    same_alone_as_among_others(few_samples(ref), pick, depth_network(START), precision=precision, rtol=rtol, max_depth=44)


@pytest.mark.parametrize("precision", [g.GCV_MIXED, g.GCV_PLAIN_FP64])
def test_trees_near_the_limit(precision, gpu_lib):
    ref = Cusps(200, 4, seed=22)
    eps = 2.0 ** -52 if precision == g.GCV_PLAIN_FP64 else 2.0 ** -46
    leaves = np.array([ref.walk(i, 1e-12, 44, eps)[1] for i in range(200)])
    pick = np.flatnonzero((leaves >= 94) & (leaves <= 127))
    assert np.sum((leaves > 96) & (leaves <= 127)) >= 30
    same_alone_as_among_others(few_samples(ref), pick, precision=precision, rtol=1e-12, max_depth=44)


@pytest.mark.parametrize("network", [None, START])
@pytest.mark.parametrize("precision", [g.GCV_MIXED, g.GCV_PLAIN_FP64])
def test_panels_are_counted_once(precision, network, gpu_lib):
    """The panel count is the tables': of 500 copies in random order 500 times one copy's, each curve by itself."""
    ref = Cusps(300, 3, seed=23)
    kw = dict(precision=precision, rtol=1e-6 if network else 1e-12, max_depth=44)
    weights = None if network is None else depth_network(network)
    b = few_samples(ref)
    alone = [table(b.subset(np.array([i])), weights, **kw)[2] for i in range(b.n_curve)]
    order = np.random.default_rng(8).permutation(np.repeat(np.arange(b.n_curve), 500))
    st = table(b.subset(order), weights, **kw)[2]
    for what in ("n_panels", "n_leaves", "n_capped", "n_deep_segments"):
        assert st[what] == 500 * sum(a[what] for a in alone), what
