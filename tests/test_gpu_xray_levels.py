"""The float-float smoothing and spline of downsample_image at the edges of its
chunks and ranges, against the oracle's double arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _image(shape, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:shape[0], 0:shape[1]]
    return (3.0 + np.sin(y / 9.0) * np.cos(x / 7.0) + 0.2 * rng.standard_normal(shape)).astype(np.float32)


# lines below, at and just above one chunk (64) and two, outputs that hardly shrink
@pytest.mark.parametrize("shape", [(63, 80), (64, 64), (65, 129), (127, 66), (192, 193)])
@pytest.mark.parametrize("factor", [0.125, 0.3, 0.5, 0.9, 0.99])
def test_levels_match_the_oracle(xr, oracle, shape, factor):
    from xreg_gb300 import api
    img = _image(shape, shape[0])
    got, ref = api.downsample_image(img, factor), oracle.downsample_image(img, factor)
    assert got.shape == ref.shape
    # both round the same double-precision value to float, within an ulp of the largest
    np.testing.assert_allclose(got, ref, rtol=0, atol=2.0 ** -23 * np.abs(ref).max())


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3e38, 2e-39])
def test_values_beyond_float_float(xr, oracle, value):
    from xreg_gb300 import api
    img = _image((150, 97), 1)
    img[70, 40] = value
    if value == 2e-39:
        img *= 1e-38
    got, ref = api.downsample_image(img, 0.5), oracle.downsample_image(img, 0.5)
    ok = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(got), ok)
    np.testing.assert_allclose(got[ok], ref[ok], rtol=2.0 ** -22, atol=2.0 ** -22 * np.abs(img[np.isfinite(img)]).max())


def test_blank_image_log_remap_and_levels(xr, oracle):
    from xreg_gb300 import api
    img = np.zeros((100, 90), np.float32)
    np.testing.assert_array_equal(api.downsample_image(img, 0.25), 0.0)
    img = _image((130, 140), 2) * 1e4
    img[5, 7] = np.inf
    np.testing.assert_array_equal(api.log_remap(img), oracle.log_remap(img))
