"""Grad-NCC at the edges of its tiles (strips of 26, 28 or 30 columns by 32 rows)
against the oracle, masked and not, and through an objective of several views."""
import numpy as np
import pytest

from tests.helpers import small_camera, small_volume
from xreg_gb300 import synth

pytestmark = pytest.mark.gpu


def _device_metric(xr, fixed, movs, smooth, mask):
    import torch
    d = torch.from_numpy(movs).cuda()
    torch.cuda.synchronize()
    m = xr.ImgSimMetric2DGradNCCCUDA()
    m.set_fixed_image(fixed)
    if mask is not None:
        m.set_mask(mask)
    m.set_smooth_img_before_sobel_kernel_radius(smooth)
    m.set_num_moving_images(len(movs))
    m.set_mov_imgs_device_buf(d.data_ptr())
    m.allocate_resources()
    m.compute()
    return m.sim_vals()


@pytest.mark.parametrize("smooth", [0, 3, 5])
@pytest.mark.parametrize("shape", [(8, 8), (31, 27), (32, 26), (33, 53), (64, 52), (65, 60), (97, 57), (130, 105)])
def test_tile_edges(xr, oracle, shape, smooth):
    rng = np.random.default_rng(shape[0] + smooth)
    fixed = rng.random(shape).astype(np.float32)
    movs = (rng.random((3,) + shape) + fixed).astype(np.float32)
    mask = (rng.random(shape) < 0.7).astype(np.uint8)
    for k in (None, mask):
        got = _device_metric(xr, fixed, movs, smooth, k)
        np.testing.assert_allclose(got, oracle.grad_ncc(fixed, movs, smooth_ksize=smooth, mask=k), atol=1e-5, rtol=0)


def test_objective_and_metric_agree(xr, oracle):
    """The batched launch of an objective gives each view's own metric values, also
    when its population, its mask or its stream changes between calls."""
    import torch
    from xreg_gb300.api import CameraModel
    vol, det = small_volume(3, (40, 36, 44)), (70, 57)
    cams = [small_camera(det, 3.0), CameraModel(small_camera(det, 3.0).desc)]
    rc = xr.RayCasterLineIntCUDA()
    rc.set_volume(vol)
    rc.set_camera_models(cams)
    rc.set_ray_step_size(0.5)
    rng = np.random.default_rng(1)
    fixed = [rng.random(det).astype(np.float32) for _ in cams]
    ms = []
    for f in fixed:
        m = xr.ImgSimMetric2DGradNCCCUDA()
        m.set_fixed_image(f)
        ms.append(m)
    obj = xr.PopulationObjective(rc, ms, 9)
    poses = synth.sample_poses(vol, synth.gt_pose(vol), 9, 8.0, 8.0, seed=5)
    stream = torch.cuda.Stream()
    for n, masked, s in ((9, False, 0), (9, False, 0), (4, False, 0), (4, True, 0), (9, True, stream.cuda_stream), (9, True, 0)):
        rc.set_stream(s)
        mask = (rng.random(det) < 0.8).astype(np.uint8) if masked else None
        for m in ms:
            m.set_mask(mask)
            m.allocate_resources()
        got = obj.eval(poses[:n])
        imgs = rc.projs()
        want = np.mean([oracle.grad_ncc(f, imgs[v * n:(v + 1) * n], mask=mask) for v, f in enumerate(fixed)], axis=0)
        np.testing.assert_allclose(got, want, atol=1e-5, rtol=0)
        np.testing.assert_array_equal(obj.eval(poses[:n]), got)
