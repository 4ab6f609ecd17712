"""The FP16 cell blend as the kernel forms it now (interp8_h16 in xr_raycast.cu):
fractions of positions in units of 2^-15 voxel, both weights of an axis from one
conversion, and the z level as b0 + fz (b1 - b0) in float.  Restated operation by
operation; the x and y levels are those of tests/test_fp16_blend_cpu.py."""
import numpy as np

from tests.test_fp16_blend_cpu import _blend_h16, _cells, _half, _hfma, _hmul, _trilinear

F, D = np.float32, np.float64


def _levels(v, fx, fy):
    """b0, b1: the x and y levels, times 2^30, in float."""
    sx, sy = F(fx * 2.0 ** 15), F(fy * 2.0 ** 15)
    FX, GX, FY, GY = _half(sx), _half(F(32768.0) - sx), _half(sy), _half(F(32768.0) - sy)
    a0 = [_hfma(v[..., 2 + z], FX, _hmul(v[..., 0 + z], GX)) for z in (0, 1)]
    a1 = [_hfma(v[..., 6 + z], FX, _hmul(v[..., 4 + z], GX)) for z in (0, 1)]
    return [F(F(a0[z].astype(D) * GY.astype(D)).astype(D) + a1[z].astype(D) * FY.astype(D)) for z in (0, 1)]


def _blend_now(v, fx, fy, fz):
    b0, b1 = _levels(v, fx, fy)
    d = F(b1 - b0)
    return F(b0.astype(D) + d.astype(D) * F(fz).astype(D)) / F(2.0 ** 30), b0, b1


def test_z_level_by_difference_within_bound():
    for seed in (3, 5):
        v, f, tiny = _cells(seed)
        f = f.copy()
        # z fractions down to and up to an ulp of a position from 0 and 1 too
        n = len(f) // 4
        f[:n, 2] = 2.0 ** -np.random.default_rng(seed).integers(7, 24, n).astype(D)
        f[n:2 * n, 2] = 1.0 - f[:n, 2]
        got, b0, b1 = _blend_now(v, f[:, 0], f[:, 1], f[:, 2])
        ref = _trilinear(v, f[:, 0], f[:, 1], f[:, 2])
        top = np.maximum(np.abs(b0), np.abs(b1)).astype(D) / 2.0 ** 30
        # four roundings to half in a row (x weight, x product, x sum, y weight) of 2^-11
        # each, and the float roundings of b1 - b0 and of the result: 2^-24 of the larger each
        bound = ref * ((1 + 2.0 ** -11) ** 4 - 1) + top * 2.0 ** -22
        assert np.all(np.abs(got.astype(D) - ref) <= bound)
        nz = ref > 0
        assert np.mean(np.abs(got.astype(D) - ref)[nz] / ref[nz]) <= 3e-4
        assert np.all(got[~nz] == 0.0)
        # against the form by weights: the same but for those two float roundings
        old = _blend_h16(v, f[:, 0], f[:, 1], f[:, 2]).astype(D)
        assert np.all(np.abs(got.astype(D) - old) <= top * 2.0 ** -22)


def test_grazing_samples_stay_exact_in_z():
    """A far z level of zeros: b1 - b0 = -b0 exactly, so the sample is b0 (1 - fz) with one rounding."""
    v, f, _ = _cells(6)
    v = v.copy()
    v[:, 1::2] = 0
    got, b0, b1 = _blend_now(v, f[:, 0], f[:, 1], f[:, 2])
    assert np.all(b1 == 0)
    want = b0.astype(D) * (1.0 - F(f[:, 2]).astype(D)) / 2.0 ** 30
    assert np.all(np.abs(got.astype(D) - want) <= np.abs(want) * 2.0 ** -24)
