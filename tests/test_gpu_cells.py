"""Sampling from the cell copy at its edges: border cells, slabs around the size
where the round-down floor constants start, volumes whose corner differences
would not be finite.  Every layout gives the same bits, within the DRR
tolerances of tests/test_gpu_drr.py of the oracle."""
import numpy as np
import pytest

from tests.helpers import drr_rel_err, oracle_cams, oracle_geom, small_camera
from xreg_gb300 import api, synth
from xreg_gb300.se3 import euler_xyz, rigid

pytestmark = pytest.mark.gpu

TOL = {0: 1e-4, 1: 2e-3, 2: 2.0 ** -8}


def _poses(vol, seed):
    """Random views, views along each axis (rays in the planes of voxels) and a half turn."""
    gt = synth.gt_pose(vol)
    C = vol.xform_img_center_to_itk_phys()
    turned = [C @ rigid(euler_xyz(*np.radians(a)), np.zeros(3)) @ np.linalg.inv(C) @ gt
              for a in ((0.0, 0.0, 0.0), (90.0, 0.0, 0.0), (0.0, 90.0, 0.0), (0.0, 0.0, 180.0), (30.0, 50.0, 10.0))]
    return np.concatenate([synth.sample_poses(vol, gt, 3, 20.0, 5.0, seed=seed), np.stack(turned)])


def _images(xr, vol, cam, poses, vt):
    """The images of each layout and loop, skipping on and off."""
    rc = xr.RayCasterLineIntCUDA()
    rc.set_volume(vol, vt)
    rc.set_camera_model(cam)
    rc.set_ray_step_size(0.5)
    rc.set_num_projs(len(poses))
    rc.allocate_resources()
    rc.distribute_xforms_among_cam_models(poses)
    out = []
    for skip in (True, False):
        rc.set_empty_space_skipping(skip)
        for layout in ((-1, 0, 1, 2, 3) if vt == 0 else (-1, 0, 1)):
            for loop in (2, 4):
                rc.set_launch_config(layout, 1, loop, 8)
                rc.compute()
                out.append(rc.projs())
    return out


# slabs of (nx + 1) x (nz + 1) cells just below and above 2^10, odd and smallest sizes
@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("size", [(2, 2, 2), (31, 5, 30), (31, 40, 31), (9, 33, 120), (65, 17, 22)])
def test_values_up_to_the_faces(xr, oracle, size, vt):
    rng = np.random.default_rng(sum(size))
    vol = api.Volume(rng.uniform(0.5, 1.0, size[::-1]).astype(np.float32), spacing=(2.0, 1.5, 1.75))
    cam, poses = small_camera((45, 37), 4.0), _poses(vol, 3)
    imgs = _images(xr, vol, cam, poses, vt)
    for img in imgs[1:]:
        np.testing.assert_array_equal(img, imgs[0])
    ref = oracle.drr_f32(vol.voxels, oracle_geom(vol), oracle_cams([cam]), poses, step=0.5)
    assert np.any(ref != 0)
    rel, zero = drr_rel_err(imgs[0], ref)
    assert zero == 0.0 and rel <= TOL[vt], rel


def test_subnormal_bf16_voxels(xr):
    """Rays that meet only voxels below 2^-126: every layout gives the same bits."""
    rng = np.random.default_rng(11)
    v = np.zeros((40, 36, 33), np.float32)
    v[6:34, 6:30, 6:15] = rng.uniform(0.5, 1.0, (28, 24, 9))
    v[6:34, 6:30, 15:27] = rng.uniform(0.0, 1.0, (28, 24, 12)) * 1e-38
    vol = api.Volume(v, spacing=(1.5, 1.5, 1.5))
    cam, poses = small_camera((45, 37), 4.0), _poses(vol, 5)
    imgs = _images(xr, vol, cam, poses, 2)
    assert np.any((imgs[0] > 0) & (imgs[0] < 1e-30))
    for img in imgs[1:]:
        np.testing.assert_array_equal(img, imgs[0])


@pytest.mark.parametrize("vt", [0, 2])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e38])
def test_values_without_finite_differences(xr, oracle, value, vt):
    rng = np.random.default_rng(7)
    v = rng.uniform(0.5, 1.0, (33, 36, 40)).astype(np.float32)
    v[14:16, 20, 18:20] = value
    vol = api.Volume(v, spacing=(1.5, 1.5, 1.5))
    cam, poses = small_camera((45, 37), 4.0), _poses(vol, 5)[:4]
    imgs = _images(xr, vol, cam, poses, vt)
    for img in imgs[1:]:
        np.testing.assert_array_equal(img, imgs[0])
    ref = oracle.drr_f32(vol.voxels, oracle_geom(vol), oracle_cams([cam]), poses, step=0.5)
    ok = np.isfinite(ref)
    assert 0 < (~ok).sum() < 0.2 * ok.size or value == 1e38
    np.testing.assert_array_equal(np.isfinite(imgs[0]), ok)
    rel, zero = drr_rel_err(np.where(ok, imgs[0], 0.0), np.where(ok, ref, 0.0))
    assert zero == 0.0 and rel <= TOL[vt], rel


# launches on either side of the rule for the deep march (at most about 155,000
# rays): ray counts that are not multiples of a batch, and one pose of the larger
# launch alone
@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("kernel", [0, 1])
def test_small_launches_equal_large_ones(xr, vt, kernel):
    vol = synth.phantom_volume((48, 44, 40), (2.0, 2.0, 2.0), 5)
    cam = small_camera((130, 141), 2.0)
    poses = synth.sample_poses(vol, synth.gt_pose(vol), 12, 20.0, 10.0, seed=4)
    rc = xr.RayCasterLineIntCUDA()
    rc.set_volume(vol, vt)
    rc.set_camera_model(cam)
    rc.set_ray_step_size(0.3)
    rc.set_kernel_id(kernel)
    rc.set_num_projs(len(poses))
    rc.allocate_resources()
    rc.distribute_xforms_among_cam_models(poses)  # 219,960 rays
    rc.compute()
    many = rc.projs()
    rc.set_launch_config(0, 1, 4, 8)
    rc.compute()
    np.testing.assert_array_equal(rc.projs(), many)
    rc.set_launch_config(-1)
    for n in (1, 8):
        rc.set_num_projs(n)
        rc.distribute_xforms_among_cam_models(poses[3:3 + n])
        rc.compute()
        np.testing.assert_array_equal(rc.projs(), many[3:3 + n])
