"""The library's own arithmetic against exact rational and long-double results, over
the ranges its callers use, their ends, and the neighbours of powers of two.

Bounds: the reciprocal of two Newton steps in FP64 is good to a unit in the last place
(2^-52), a float-float reciprocal to 2^-45 (one Newton step in FP32, its input and result
rounded to 48 bits); conversions and scalings are exact where the result has the digits.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="session")
def apply(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    tmp = tmp_path_factory.mktemp("arith")
    exe = str(tmp / "arith_driver")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "gcurval_gb300", "csrc"), "-o", exe,
                        os.path.join(ROOT, "tests", "arith", "arith_driver.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def call(op, x, y=0.0):
        x = np.asarray(x, np.float64)
        fin, fout = str(tmp / "in.bin"), str(tmp / "out.bin")
        np.stack([x, np.broadcast_to(np.asarray(y, np.float64), x.shape)], 1).tofile(fin)
        r = subprocess.run([exe, str(op), fin, fout], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, (r.returncode, r.stderr)
        return np.fromfile(fout).reshape(-1, 2)

    return call


def values(lo, hi, n=200_000, seed=0):
    """Positive doubles with exponents in [lo, hi), the powers of two there and their neighbours."""
    rng = np.random.default_rng(seed)
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))
    p = np.ldexp(1.0, np.arange(lo + 1, hi))
    near = [p, np.nextafter(p, 0), np.nextafter(p, np.inf)]
    near += [p * (1 + sign * 2.0 ** -k) for k in range(20, 53) for sign in (-1, 1)]
    return np.concatenate([x] + near)


def worst(got, want):
    return float(np.max(np.abs(got.astype(np.longdouble).reshape(want.shape) / want - 1)))


def test_reciprocal(apply):
    x = values(-1000, 1000)
    assert worst(apply(0, x)[:, 0], 1 / x.astype(np.longdouble)) <= 2.0 ** -52
    ends = np.array([5e-324, 2.0 ** -1074 * 3, 2.0 ** -1022, 2.0 ** 1023, 1.7e308, np.inf])
    with np.errstate(divide="ignore", over="ignore"):
        np.testing.assert_array_equal(apply(0, ends)[:, 0], 1.0 / ends)


def test_kronrod_root_of_nothing(apply):
    assert not apply(1, [0.0, -0.0, -1.0, -1e-300, 2.0 ** -71, 5e-324]).any()


def test_float_float_reciprocal(apply):
    x = values(-100, 100)
    assert worst(apply(4, x).astype(np.longdouble).sum(1), 1 / x.astype(np.longdouble)) <= 2.0 ** -45


def test_fixed_point(apply):
    rng = np.random.default_rng(1)
    ends = np.ldexp(rng.integers(-(1 << 48), (1 << 48) + 1, 100_000).astype(np.float64), -48)  # panel ends
    ends = np.r_[ends, -1.0, 1.0, 0.0, -0.0, 2.0 ** -60, -(2.0 ** -60), 1.0 - 2.0 ** -53]
    np.testing.assert_array_equal(apply(5, ends)[:, 0], ends)
    x = rng.uniform(-1.9, 1.9, 100_000) * 2.0 ** rng.integers(-70, 1, 100_000)
    assert np.max(np.abs(apply(5, x)[:, 0] - x)) <= 2.0 ** -52  # the result is rounded to a double again
    f = x.astype(np.float32).astype(np.float64)
    assert np.max(np.abs(apply(6, f)[:, 0] - f)) <= 2.0 ** -60


def test_scaled_conversion(apply):
    x = np.r_[values(-900, 900, seed=2), -values(-900, 900, n=1000, seed=3)]
    s = np.floor(np.log2(np.abs(x))).astype(int) + np.random.default_rng(4).integers(-60, 60, x.size)
    got = apply(7, x, s).astype(np.longdouble).sum(1)
    assert worst(got, np.ldexp(x.astype(np.longdouble), -s)) <= 2.0 ** -47
    tiny = apply(7, [1.0, -3.0, 0.0, 5e-324], [71, 80, 0, -1000])
    assert not tiny.any()
    big = apply(7, [1.0, -1.0, np.inf, -np.inf], [-127, -200, 0, 900])[:, 0]
    np.testing.assert_array_equal(big, [np.inf, -np.inf, np.inf, -np.inf])
    assert np.isnan(apply(7, [np.nan], [5])[0, 0])


def test_exponents(apply):
    x = np.r_[values(-900, 900, seed=5), -values(-900, 900, n=1000, seed=6)]
    s = np.random.default_rng(7).integers(-100, 100, x.size)
    np.testing.assert_array_equal(apply(8, x, s)[:, 0], np.ldexp(x, -s))
    np.testing.assert_array_equal(apply(8, [0.0, 1.0, 1.0, -1.0, np.inf], [5, 1023, -1024, -2000, 3])[:, 0],
                                  [0.0, 0.0, np.inf, -np.inf, np.inf])
    f = np.r_[values(-149, 127, seed=8).astype(np.float32), np.float32([0, np.inf, -np.inf, 1e-45, -3.5])].astype(np.float64)
    np.testing.assert_array_equal(apply(9, f)[:, 0], f)
    assert np.isnan(apply(9, [np.nan])[0, 0])
    d = np.array([5e-324, 3e-320, -1e-310, 0.0, 2.0 ** -1022, 1.0])
    lifted = apply(10, d, 7)
    np.testing.assert_array_equal(lifted[:, 0], np.where(np.abs(d) < 2.0 ** -1022, d * 2.0 ** 64, d))
    np.testing.assert_array_equal(lifted[:, 1], np.where(np.abs(d) < 2.0 ** -1022, 71, 7))
    y, down = np.array([1.5, 1.0, 1.0, 1.0, -3.0, 1.0, 1.0, 0.0]), np.array([3, 252, -252, -100, -5, 400, -400, 17])
    np.testing.assert_array_equal(apply(11, y, down)[:, 0], [0.1875, 0.0, np.inf, 2.0 ** 100, -96.0, 0.0, np.inf, 0.0])
