"""Levels of fixed images: the float-float smoothing and spline give the floats that the
oracle's double arithmetic gives, and images with values that float-float does not
carry take the double spline, spread over lines longer than its launch has threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _image(shape, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:shape[0], 0:shape[1]]
    return (3.0 + np.sin(y / 9.0) * np.cos(x / 7.0) + 0.2 * rng.standard_normal(shape)).astype(np.float32)


@pytest.mark.parametrize("factor", [0.125, 0.25, 0.5, 0.9])
@pytest.mark.parametrize("kind", ["log", "counts"])
def test_levels_are_the_double_result(xr, oracle, factor, kind):
    from xreg_gb300 import api
    img = _image((517, 631), 3)
    if kind == "counts":
        img = np.round(4e4 * np.exp(-np.abs(img))).astype(np.float32)
    got, ref = api.downsample_image(img, factor), oracle.downsample_image(img, factor)
    # Two results that round the same value and differ by 2^-44 of it before rounding
    # (float-float) fall on two floats for 2^-44 / 2^-25 = 2^-19 of all values, then by
    # one spacing; the smoothed image, rounded once before, can add as much again for
    # each of the 4 x 4 coefficients that weigh in an output.
    assert np.mean(got != ref) <= 17 * 2.0 ** -19 + 2.0 / got.size
    np.testing.assert_allclose(got, ref, rtol=2.0 ** -23, atol=2.0 ** -23 * np.abs(ref).max() * np.any(got != ref))


@pytest.mark.parametrize("shape,factor", [((64, 3000), 0.125), ((3000, 64), 0.125), ((700, 90), 0.3), ((130, 1100), 0.5)])
@pytest.mark.parametrize("value", [np.nan, np.inf, 3e38])
def test_values_beyond_float_float_on_long_lines(xr, oracle, shape, factor, value):
    from xreg_gb300 import api
    img = _image(shape, 1)
    img[shape[0] // 2, shape[1] - 7] = value
    got, ref = api.downsample_image(img, factor), oracle.downsample_image(img, factor)
    ok = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(got), ok)
    # both in double: the same value to rounding
    np.testing.assert_allclose(got[ok], ref[ok], rtol=2.0 ** -22, atol=2.0 ** -22 * np.abs(img[np.isfinite(img)]).max())
