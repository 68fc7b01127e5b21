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
