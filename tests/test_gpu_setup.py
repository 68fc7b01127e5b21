"""Set-up of knot intervals (power-basis coefficients by the polar form) where it
can go wrong: every degree and dimension, in FP64 and in float-float, spans much
shorter than their neighbours, knots of full and of single multiplicity, knots far
from unit scale and far from the origin.

The reference is the curve itself in NumPy: de Boor's recursion for the derivative
in long double, 40 Gauss points in each knot interval after 6 dyadic cuts.  The
curves are smooth and bend little (control points close to a line), so the
reference's own error is far below the tolerances: 1e-12 for FP64 at rtol 1e-12
(the walk's tolerance, rounding well below it), 1e-11 for mixed at rtol 1e-12
(float-float coefficients, 2^-47 each over at most 30 steps, times a condition
number of at most 4 for the derivative of such curves).
"""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu

X40, W40 = np.polynomial.legendre.leggauss(40)


def knots_of(kind, p, rng):
    """A clamped vector on [0, 1] of ten inner knots, or fewer when they repeat."""
    inner = np.sort(rng.uniform(0.05, 0.95, 10))
    if kind == "short":          # spans of 1e-7 and 1e-5 beside ones of about 0.1
        inner[3], inner[7] = inner[2] + 1e-7, inner[6] + 1e-5
    elif kind == "repeated":     # multiplicity p (a corner) and, where p allows it, 2
        inner = np.sort(np.r_[inner[:4], [inner[5]] * p, [inner[8]] * min(2, p)])
    elif kind == "unclamped":
        return np.linspace(0.0, 1.0, 12 + p)
    return np.r_[np.zeros(p + 1), inner, np.ones(p + 1)]


def length(p, d, knots, ctrl):
    """Length over [k_p, k_{n-p-1}] in long double."""
    k = knots.astype(np.longdouble)
    c = ctrl.reshape(-1, d).astype(np.longdouble)
    n = len(c)
    q = np.zeros((n - 1, d), np.longdouble)
    for j in range(n - 1):
        if k[j + p + 1] > k[j + 1]:
            q[j] = p * (c[j + 1] - c[j]) / (k[j + p + 1] - k[j + 1])
    total = np.longdouble(0)
    for s in range(p, n):
        if not k[s + 1] > k[s]:
            continue
        edges = k[s] + (k[s + 1] - k[s]) * np.arange(65, dtype=np.longdouble) / 64
        mid, hw = (edges[1:] + edges[:-1]) / 2, (edges[1:] - edges[:-1]) / 2
        u = (mid[:, None] + hw[:, None] * X40).ravel()
        w = (hw[:, None] * W40).ravel()
        b = [np.broadcast_to(q[s - p + i], (u.size, d)) for i in range(p)]  # degree p-1 on knots k[1:-1]
        for r in range(1, p):
            for i in range(p - 1, r - 1, -1):
                lo, hi = k[s - p + 1 + i], k[s + 1 + i - r]
                a = ((u - lo) / (hi - lo))[:, None]
                b[i] = (1 - a) * b[i - 1] + a * b[i]
        total += (w * np.sqrt((b[p - 1] ** 2).sum(1))).sum()
    return float(total)


@pytest.mark.parametrize("precision", [g.GCV_PLAIN_FP64, g.GCV_MIXED])
@pytest.mark.parametrize("kind,scale,shift", [("plain", 1.0, 0.0), ("short", 1.0, 0.0), ("repeated", 1.0, 0.0),
                                              ("unclamped", 1.0, 0.0), ("plain", 2.0 ** 60, 0.0),
                                              ("plain", 2.0 ** -60, 0.0), ("plain", 1.0, 1000.0)])
def test_lengths_over_every_degree(precision, kind, scale, shift, gpu_lib):
    rng = np.random.default_rng(11)
    deg, dim, nk, nc, knots, ctrl, want = [], [], [], [], [], [], []
    for p in range(1, 6):
        for d in (2, 3):
            k = knots_of(kind, p, rng) * scale + shift
            n = k.size - p - 1
            c = np.c_[np.linspace(0, 1, n), 0.02 * rng.normal(size=(n, d - 1))].reshape(-1)
            want.append(length(p, d, k, c))
            deg.append(p), dim.append(d), nk.append(k.size), nc.append(c.size), knots.append(k), ctrl.append(c)
    batch = ds._pack(np.ones(len(deg)), deg, dim, nk, np.concatenate(knots), nc, np.concatenate(ctrl),
                     np.full(len(deg), 9), "setup", 1e-12)
    calc = g.ArclengthCalculateGpu.from_batch(batch, precision=precision, rtol=1e-12)
    calc.createArclengthTable()
    tol = 1e-11 if precision == g.GCV_MIXED else 1e-12
    np.testing.assert_allclose(calc.getAllCurveArclengths(), want, rtol=tol)
