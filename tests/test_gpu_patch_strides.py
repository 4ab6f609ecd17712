"""Patch metrics on both sides of the rule for the patches a thread scores: at stride 3
most tiles of four rows leave room for one block an SM only, and one row is taken
whatever the number of images.  An image alone and among many gives the same bits, and
both are within the metric tests' bound (1e-5) of the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grad", [0, 1])
@pytest.mark.parametrize("radius,stride", [(1, 3), (3, 3), (5, 3), (7, 3), (7, 2), (9, 2), (9, 3), (2, 4)])
@pytest.mark.parametrize("masked", [False, True])
def test_alone_and_among_many(xr, oracle, grad, radius, stride, masked):
    import torch
    shape, nimgs = ((203, 230) if stride == 2 else (290, 306) if stride == 3 else (387, 400)), 23
    rng = np.random.default_rng(radius * 10 + stride)
    fixed = rng.random(shape).astype(np.float32)
    movs = (0.5 * rng.random((nimgs,) + shape) + fixed).astype(np.float32)
    mask = (rng.random(shape) < 0.7).astype(np.uint8) if masked else None
    d = torch.from_numpy(movs).cuda()
    torch.cuda.synchronize()
    got = []
    for first, n in [(0, nimgs), (nimgs - 1, 1)]:
        m = (xr.ImgSimMetric2DPatchGradNCCCUDA if grad else xr.ImgSimMetric2DPatchNCCCUDA)()
        m.set_fixed_image(fixed)
        if masked:
            m.set_mask(mask)
        m.set_patch_radius(radius)
        m.set_patch_stride(stride)
        m.set_num_moving_images(n)
        m.set_mov_imgs_device_buf(d[first:].data_ptr())
        m.allocate_resources()
        m.compute()
        got.append(np.array(m.sim_vals()))
    assert nimgs * ((shape[0] - 2 * radius) // stride) * ((shape[1] - 2 * radius) // stride) > 152 * 1024
    np.testing.assert_array_equal(got[1], got[0][-1:])
    f = oracle.patch_grad_ncc_ex if grad else oracle.patch_ncc_ex
    ref = f(fixed, movs[[0, -1]], radius=radius, stride=stride, mask=mask)
    np.testing.assert_allclose(got[0][[0, -1]], ref, atol=1e-5, rtol=0)


@pytest.mark.parametrize("masked,nimgs", [(False, 1), (False, 60), (True, 1), (True, 60)])
def test_the_largest_windows_are_refused_alike(xr, masked, nimgs):
    """Both gradients' tile of 16 x 16 patches must fit 200 KB, whatever kernel runs."""
    import torch
    from xreg_gb300 import XRegError
    shape = (150, 170)
    rng = np.random.default_rng(4)
    d = torch.from_numpy(rng.random((nimgs,) + shape).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    for radius, stride, ok in [(10, 4, True), (11, 4, False), (12, 4, False), (16, 3, True), (16, 4, False)]:
        m = xr.ImgSimMetric2DPatchGradNCCCUDA()
        m.set_fixed_image(rng.random(shape).astype(np.float32))
        if masked:
            m.set_mask((rng.random(shape) < 0.7).astype(np.uint8))
        m.set_patch_radius(radius)
        m.set_patch_stride(stride)
        m.set_num_moving_images(nimgs)
        m.set_mov_imgs_device_buf(d.data_ptr())
        m.allocate_resources()
        if ok:
            m.compute()
            assert np.all(np.isfinite(m.sim_vals()))
        else:
            with pytest.raises(XRegError):
                m.compute()
