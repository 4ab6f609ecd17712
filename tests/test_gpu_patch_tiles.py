"""Patch metrics at the edges of their tiles (32 columns by 8 or 32 rows of patches,
images in pairs), masked and not, every stride, against the oracle; the same bounds
as the other metric tests (1e-5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# patch grids of 31, 32, 33, 64 and 65 rows or columns at radius 5, odd leftovers
@pytest.mark.parametrize("grad", [0, 1])
@pytest.mark.parametrize("shape,radius,stride", [((41, 42), 5, 1), ((43, 75), 5, 1), ((74, 43), 5, 1), ((75, 53), 5, 1),
                                                 ((73, 75), 5, 2), ((140, 75), 5, 2), ((60, 111), 3, 3), ((70, 67), 2, 4),
                                                 ((40, 39), 1, 1), ((50, 47), 7, 1)])
@pytest.mark.parametrize("masked,nimgs", [(False, 3), (True, 3), (False, 1)])
def test_tile_edges(xr, oracle, grad, shape, radius, stride, masked, nimgs):
    import torch
    rng = np.random.default_rng(shape[0] * 7 + stride)
    fixed = rng.random(shape).astype(np.float32)
    movs = (0.5 * rng.random((nimgs,) + shape) + fixed).astype(np.float32)
    d = torch.from_numpy(movs).cuda()
    torch.cuda.synchronize()
    m = (xr.ImgSimMetric2DPatchGradNCCCUDA if grad else xr.ImgSimMetric2DPatchNCCCUDA)()
    m.set_fixed_image(fixed)
    mask = None
    if masked:
        mask = (rng.random(shape) < 0.7).astype(np.uint8)
        m.set_mask(mask)
    m.set_patch_radius(radius)
    m.set_patch_stride(stride)
    m.set_num_moving_images(nimgs)
    m.set_mov_imgs_device_buf(d.data_ptr())
    m.allocate_resources()
    m.compute()
    f = oracle.patch_grad_ncc_ex if grad else oracle.patch_ncc_ex
    np.testing.assert_allclose(m.sim_vals(), f(fixed, movs, radius=radius, stride=stride, mask=mask), atol=1e-5, rtol=0)


@pytest.mark.parametrize("grad", [0, 1])
@pytest.mark.parametrize("radius,stride", [(5, 1), (5, 2), (3, 3)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_masked_out_pixel_that_is_not_finite(xr, grad, radius, stride, bad):
    """Masked-out pixels take no part in a patch's sum: a patch with no other pixels
    scores 1, whatever they hold, and patches without the pixel are not touched."""
    import torch
    rng = np.random.default_rng(3)
    fixed = rng.random((48, 60)).astype(np.float32)
    movs = (0.5 * rng.random((3, 48, 60)) + fixed).astype(np.float32)
    mask = np.ones((48, 60), np.uint8)
    mask[:, :30] = 0
    scores = []
    for v in (0.25, bad):
        movs[:, 5, 5] = v
        d = torch.from_numpy(movs.copy()).cuda()
        torch.cuda.synchronize()
        m = (xr.ImgSimMetric2DPatchGradNCCCUDA if grad else xr.ImgSimMetric2DPatchNCCCUDA)()
        m.set_fixed_image(fixed)
        m.set_mask(mask)
        m.set_patch_radius(radius)
        m.set_patch_stride(stride)
        m.set_patch_options(use_mask_for_weighting=0, weight_patch_sims_in_combine=0, save_all_per_patch_scores=1)
        m.set_num_moving_images(3)
        m.set_mov_imgs_device_buf(d.data_ptr())
        m.allocate_resources()
        m.compute()
        scores.append(np.stack([m.patch_scores(i) for i in range(3)]))
    np.testing.assert_array_equal(scores[1], scores[0])
    assert (scores[1] == 1.0).any()


@pytest.mark.parametrize("grad", [0, 1])
@pytest.mark.parametrize("shape,radius,stride,masked,nimgs", [((200, 331), 5, 1, False, 33), ((200, 331), 5, 1, True, 33),
                                                              ((97, 140), 3, 1, False, 41), ((253, 210), 5, 2, True, 41),
                                                              ((253, 210), 5, 2, False, 41)])
def test_an_image_alone_or_among_many(xr, grad, shape, radius, stride, masked, nimgs):
    """Few patches are scored one a thread, many four: the same bits."""
    import torch
    rng = np.random.default_rng(shape[0])
    fixed = rng.random(shape).astype(np.float32)
    movs = (0.5 * rng.random((nimgs,) + shape) + fixed).astype(np.float32)
    d = torch.from_numpy(movs).cuda()
    torch.cuda.synchronize()
    got = []
    for first, n in [(0, nimgs), (0, 1), (nimgs - 1, 1), (3, 2)]:
        m = (xr.ImgSimMetric2DPatchGradNCCCUDA if grad else xr.ImgSimMetric2DPatchNCCCUDA)()
        m.set_fixed_image(fixed)
        if masked:
            m.set_mask((np.arange(movs[0].size).reshape(shape) % 7 != 0).astype(np.uint8))
        m.set_patch_radius(radius)
        m.set_patch_stride(stride)
        m.set_num_moving_images(n)
        m.set_mov_imgs_device_buf(d[first:].data_ptr())
        m.allocate_resources()
        m.compute()
        got.append((first, np.array(m.sim_vals())))
    for first, v in got[1:]:
        np.testing.assert_array_equal(v, got[0][1][first:first + len(v)])
