"""The warp-wide length walk where its bookkeeping can go wrong: intervals with
more leaves than a warp keeps for one interval, warps that run out of panel
nodes, batches smaller and larger than a warp's claim, capped depths, and
results that do not depend on how the work was shared out.

Curves: degree-5 pieces whose derivative vanishes at points inside the interval
(cusps), where the walk refines down to its tolerance on both sides.  The
reference is the walk itself in NumPy: the same panels, rule and acceptance test
in FP64 (an independent integral is no reference here: any adaptive rule can
accept a panel with a cusp inside by accident).  A panel whose error estimate
meets the tolerance within rounding may fall either way, which moves a length by
no more than the tolerance, rtol of it.
"""
from math import comb

import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu


class Cusps:
    """n planar quintic Bezier curves C' = prod (x - c_i) (q_x, q_y) on [0, 1]."""

    def __init__(self, n, cusps, seed):
        rng = np.random.default_rng(seed)
        # monomial -> Bernstein coefficients, degree 5
        m = np.array([[comb(j, i) / comb(5, i) if j >= i else 0.0 for i in range(6)] for j in range(6)])
        self.derv, self.roots, ctrl = [], [], []
        for _ in range(n):
            self.roots.append(np.sort(rng.uniform(0.1, 0.9, cusps)))
            root = np.poly1d(self.roots[-1], r=True)
            derv = [root * np.poly1d(rng.normal(size=5 - cusps)) for _ in range(2)]
            self.derv.append(derv)
            pts = []
            for p in derv:
                c = np.zeros(6)
                a = np.polyint(p).c[::-1]
                c[:a.size] = a
                pts.append(m @ c)
            ctrl.append(np.stack(pts, 1).reshape(-1))
        knots = np.tile(np.repeat([0.0, 1.0], 6), n)
        self.batch = ds._pack(np.ones(n), np.full(n, 5), np.full(n, 2), np.full(n, 12), knots, np.full(n, 12),
                              np.concatenate(ctrl), np.full(n, 23), "cusps", 1e-10)

    def walk(self, i, rtol, max_depth, eps):
        """(length, leaves, capped) of curve i by depth-first G7-K15 bisection of v in [-1, 1]."""
        x, wk, wg = GK
        fx, fy = self.derv[i]

        def panel(k, depth):
            hw = 2.0 ** -depth
            v = -1.0 + (2 * k + 1) * hw + hw * x
            f = 0.5 * np.hypot(fx(0.5 * (v + 1)), fy(0.5 * (v + 1)))
            return hw * (wk @ f), hw * (wg @ f)

        total, leaves, capped = 0.0, 0, 0
        todo = [(0, 0)]
        while todo:
            k, depth = todo.pop()
            K, G = panel(k, depth)
            if depth == 0:
                tol = rtol * abs(K)
            ok = abs(K - G) <= max(tol * 2.0 ** -depth, 50 * eps * abs(K))
            if ok or depth >= max_depth:
                total, leaves, capped = total + K, leaves + 1, capped + (not ok)
            else:
                todo += [(2 * k + 1, depth + 1), (2 * k, depth + 1)]
        return total, leaves, capped


# G7-K15: nodes, Kronrod weights, Gauss weights (zero on the Kronrod-only nodes)
_X = [0.991455371120812639206854697526329, 0.949107912342758524526189684047851, 0.864864423359769072789712788640926,
      0.741531185599394439863864773280788, 0.586087235467691130294144845693013, 0.405845151377397166906606412076961,
      0.207784955007898467600689403773245]
_WK = [0.022935322010529224963732008058970, 0.063092092629978553290700663189204, 0.104790010322250183839876322541518,
       0.140653259715525918745189590510238, 0.169004726639267902826583426598550, 0.190350578064785409913256402421014,
       0.204432940075298892414161999234649]
_WG = [0.0, 0.129484966168869693270611432679082, 0.0, 0.279705391489276667901467771423780, 0.0,
       0.381830050505118944950369775488975, 0.0]
GK = (np.array([-v for v in _X] + [0.0] + _X[::-1]),
      np.array(_WK + [0.209482141084727828012999174891714] + _WK[::-1]),
      np.array(_WG + [0.417959183673469387755102040816327] + _WG[::-1]))


def build(b, **kw):
    calc = g.ArclengthCalculateGpu.from_batch(b, collect_stats=True, **kw)
    calc.createArclengthTable()
    return calc


@pytest.mark.parametrize("precision,rtol", [(g.GCV_PLAIN_FP64, 1e-12), (g.GCV_PLAIN_FP64, 1e-9), (g.GCV_MIXED, 1e-8),
                                            (g.GCV_MIXED, 1e-11)])
@pytest.mark.parametrize("n,cusps", [(1, 3), (3, 2), (9, 0), (33, 3), (700, 3)])
def test_cusps(n, cusps, precision, rtol, gpu_lib):
    ref = Cusps(n, cusps, seed=n)
    b = ref.batch
    calc = build(b, precision=precision, rtol=rtol, max_depth=44)
    eps = 2.0 ** -52 if precision == g.GCV_PLAIN_FP64 else 2.0 ** -46
    want = np.array([ref.walk(i, rtol, 44, eps) for i in range(n)])
    L = calc.getAllCurveArclengths()
    assert np.max(np.abs(L - want[:, 0]) / want[:, 0]) <= rtol + 1e-13
    leaves = want[:, 1].sum()
    assert abs(calc.stats()["n_leaves"] - leaves) <= 0.002 * leaves + 1
    u = calc.arclengthReverse(b.n_samples, b.sample_positions(), True, g.GCV_HOST).us.reshape(n, -1)
    assert np.all(np.diff(u, axis=1) >= 0.0) and np.all(u[:, 0] == 0.0) and np.all(u[:, -1] == 1.0)
    # another build, another sharing-out of the work: the same numbers
    calc.createArclengthTable()
    np.testing.assert_array_equal(calc.getAllCurveArclengths(), L)


def test_deep_list_takes_what_a_warp_does_not_keep(gpu_lib):
    ref = Cusps(64, 3, seed=5)
    leaves = np.array([ref.walk(i, 1e-12, 44, 2.0 ** -52)[1] for i in range(64)])
    st = build(ref.batch, precision=g.GCV_PLAIN_FP64, rtol=1e-12, max_depth=44).stats()
    assert abs(st["n_deep_segments"] - np.sum(leaves > 96)) <= np.sum(np.abs(leaves - 96) <= 2)
    assert np.sum(leaves > 96) > 0


@pytest.mark.parametrize("max_depth", [1, 4, 44, 48])
@pytest.mark.parametrize("precision", [g.GCV_PLAIN_FP64, g.GCV_MIXED])
def test_depth_cap(precision, max_depth, gpu_lib):
    b = Cusps(40, 2, seed=8).batch
    st = build(b, precision=precision, rtol=1e-9, max_depth=max_depth).stats()
    assert st["n_leaves"] <= 40 * 2 ** min(max_depth, 20)
    assert (st["n_capped"] > 0) == (max_depth <= 4)


@pytest.mark.parametrize("network", [False, True])
def test_work_sharing_does_not_change_the_table(network, gpu_lib):
    """Builds with the launch shapes the tuner tries (other claims per warp) and with a fresh leaf pool."""
    b = ds.uneven_batch(900, seed=61, max_ctrl=300, max_samples=32)
    out = []
    for _ in range(2):
        calc = g.ArclengthCalculateGpu.from_batch(b, precision=g.GCV_MIXED, rtol=1e-9, learned=network)
        if network:
            from gcurval_gb300 import learned
            calc.set_learned_model(learned.load_model())
        for _ in range(4):
            calc.createArclengthTable()
            out.append((calc.getAllCurveArclengths(),
                        calc.arclengthReverse(b.n_samples, b.sample_positions(), True, g.GCV_HOST).us))
        calc.close()
    for L, u in out[1:]:
        np.testing.assert_array_equal(L, out[0][0])
        np.testing.assert_array_equal(u, out[0][1])


@pytest.mark.parametrize("rtol,max_depth", [(1e-9, 30), (1e-12, 44), (1e-12, 45), (0.9e-12, 44), (1e-9, 3)])
@pytest.mark.parametrize("n", [1, 5, 300])
def test_lengths_without_a_table(n, rtol, max_depth, gpu_lib):
    """gcv_bspline_lengths_noalloc on both sides of its rule, against the walk in NumPy."""
    import ctypes

    torch = pytest.importorskip("torch")
    ref = Cusps(n, 3, seed=n + 1)
    b = ref.batch
    ko = torch.from_numpy(b.knot_off.astype(np.int32)).cuda()
    kv, cp = torch.from_numpy(b.knots).cuda(), torch.from_numpy(b.ctrl).cuda()
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    capped = ctypes.c_int64()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert gpu_lib.gcv_bspline_lengths_noalloc(n, 5, 2, p(ko), p(kv), p(cp), rtol, max_depth, p(out), None,
                                               ctypes.byref(capped)) == 0
    want = np.array([ref.walk(i, rtol, max_depth, 2.0 ** -52) for i in range(n)])
    assert np.max(np.abs(out.cpu().numpy() - want[:, 0]) / want[:, 0]) <= rtol + 1e-13
    assert abs(capped.value - want[:, 2].sum()) <= 0.002 * want[:, 2].sum()
