"""Parameters of curves whose knots are far smaller than 1: scaled by a power of two
they are those of the unscaled knots (twice the sampler's stopping threshold apart at
most, a tenth of rtol each, over a speed of at least half the length per knot range)."""
import numpy as np
import pytest

import gcurval_gb300 as g
from test_gpu_knot_units import curves, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rtol", [1e-10, 1e-12, 0.9e-12])
@pytest.mark.parametrize("precision,power", [(g.GCV_PLAIN_FP64, -900), (g.GCV_PLAIN_FP64, -980), (g.GCV_PLAIN_FP64, -1000),
                                             (g.GCV_PLAIN_FP64, 1000), (g.GCV_MIXED, -100), (g.GCV_MIXED, 100)])
def test_parameters_scale_with_the_knots(precision, power, rtol, gpu_lib):
    _, u0, _ = run(curves(0, 0), precision, rtol)
    _, u, _ = run(curves(power, 0), precision, rtol)
    np.testing.assert_allclose(u * 2.0 ** -power, u0, rtol=0, atol=max(0.4 * rtol, 1e-14))
