"""Semi-axes of either sign and of very different magnitudes: the length and the
samples depend on their squares only, so they are those of the positive axes."""
import numpy as np
import pytest
from scipy.special import ellipe

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu

AXES = [(-1.0, 1e-20), (-1.0, -1e-20), (1e-20, -1.0), (-1e-20, -1.0), (-3.0, -2.0), (-1e-30, 1.0), (-2.0, 0.0),
        (0.0, -2.0), (-1e150, 1e100), (-1e-100, 1e-140)]


@pytest.mark.parametrize("precision,rtol", [(g.GCV_PLAIN_FP64, 1e-10), (g.GCV_PLAIN_FP64, 1e-12),
                                            (g.GCV_PLAIN_FP64, 0.9e-12), (g.GCV_MIXED, 1e-9)])
def test_signs_of_the_axes_do_not_matter(precision, rtol, gpu_lib):
    axes = np.array([a for a in AXES if precision == g.GCV_PLAIN_FP64 or max(map(abs, a)) < 1e18 > 1e-18 < max(map(abs, a))])
    out = []
    for ab in (axes, np.abs(axes)):
        b = ds.ellipses_from_axes(ab[:, 0], ab[:, 1], n_samples=0)
        b.n_samples[:] = 17
        calc = g.ArclengthCalculateGpu.from_batch(b, precision=precision, rtol=rtol)
        calc.createArclengthTable()
        out.append((calc.getAllCurveArclengths(), calc.arclengthReverse(b.n_samples, b.sample_positions(), True, g.GCV_HOST).us))
    big, small = np.abs(axes).max(1), np.abs(axes).min(1)
    want = 4.0 * big * ellipe(1.0 - (small / big) ** 2)
    np.testing.assert_allclose(out[1][0], want, rtol=rtol)
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("rtol", [1e-10, 1e-12])
def test_axes_whose_squares_vanish(rtol, gpu_lib):
    """Semi-axes of 1e-165 and below: length 0, as the FP64 kernels (below rtol 1e-12) have it, and never NaN."""
    a = 10.0 ** -np.r_[165.0, 172, 173, 174, 180, 250, 300]
    e = ds.ellipses_from_axes(np.r_[a, -a, a], np.r_[a, a, 0.3 * a])
    for r in (rtol, 0.5e-12):
        calc = g.ArclengthCalculateGpu.from_batch(e, precision=g.GCV_PLAIN_FP64, rtol=r)
        calc.createArclengthTable()
        assert not calc.getAllCurveArclengths().any()


def test_axes_with_denormal_squares(gpu_lib):
    """Semi-axes of 1e-153 to 1e-157: the squares keep 2^-53 to 2^-28 of themselves."""
    a = 10.0 ** -np.r_[153.0, 154, 155, 156, 157]
    e = ds.ellipses_from_axes(np.r_[a, -a], np.r_[a, a])
    calc = g.ArclengthCalculateGpu.from_batch(e, precision=g.GCV_PLAIN_FP64, rtol=1e-10, max_depth=10)
    calc.createArclengthTable()
    np.testing.assert_allclose(calc.getAllCurveArclengths(), 2.0 * np.pi * np.r_[a, a], rtol=1e-8)
