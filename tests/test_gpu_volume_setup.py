"""Volume set-up: HU to attenuation at its rounding edges, the statistics pass and
the cell build at the edges of their tiles, and one volume set over another."""
import numpy as np
import pytest

from tests.helpers import drr_rel_err, oracle_cams, oracle_geom, small_camera
from xreg_gb300 import XRegError, api, synth

pytestmark = pytest.mark.gpu


def _device(a):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    torch.cuda.synchronize()
    return t


def test_hu_to_mu_is_the_double_result(xr):
    import torch
    rng = np.random.default_rng(1)
    hu = np.concatenate([rng.uniform(-1100.0, 3000.0, 2_000_003), -1000.0 + rng.exponential(1.0, 500_000) * 10.0 ** rng.integers(-5, 2, 500_000),
                         [-1000.0, np.nextafter(np.float32(-1000), np.float32(0)), -999.9999, 0.0, -0.0, 1e30, -1e30, np.inf, -np.inf, np.nan,
                          1e-40]]).astype(np.float32)
    d_hu = _device(hu)
    d_mu = torch.empty_like(d_hu)
    torch.cuda.synchronize()
    api.hu_to_lin_att_device(d_hu.data_ptr(), hu.size, d_mu.data_ptr())
    torch.cuda.synchronize()
    scale = (0.02683 - 0.02485e-4) * 1.0e-3
    with np.errstate(invalid="ignore"):
        v = (hu.astype(np.float64) * scale + 0.02683) - (-1000.0 * scale + 0.02683)
        ref = np.where(v > 0.0, v, 0.0).astype(np.float32)
    got = d_mu.cpu().numpy()
    # the product may keep more digits than numpy's (a fused multiply-add), which can
    # move a result by an ulp where the double values straddle a rounding boundary
    assert np.mean(got != ref) < 1e-6
    np.testing.assert_allclose(got, ref, rtol=2.0 ** -23, atol=0)


# edges of the build's 32 x 16 x 32 tiles, of 8^3 macro cells and of 1024-voxel row segments
@pytest.mark.parametrize("size", [(2, 2, 2), (31, 15, 32), (32, 16, 31), (33, 17, 65), (1023, 3, 9), (1033, 9, 10), (516, 9, 17), (1028, 17, 9)])
@pytest.mark.parametrize("vt,tol", [(0, 1e-4), (1, 2e-3), (2, 2.0 ** -8)])
def test_sparse_volumes(xr, oracle, size, vt, tol):
    """Few non-zero voxels, corners among them: skipping loses none of them, the
    cell copy and the voxels agree, host and device sources give the same volume."""
    rng = np.random.default_rng(sum(size) + vt)
    v = np.zeros(size[::-1], np.float32)
    for z, y, x in [(0, 0, 0), (-1, -1, -1), (0, -1, 0), (-1, 0, -1)] + [tuple(rng.integers(0, n) for n in v.shape) for _ in range(6)]:
        v[z, y, x] = rng.uniform(0.5, 1.0)
    vol = api.Volume(v, spacing=(1.0, 1.0, 1.0) if size[0] < 500 else (0.2, 6.0, 6.0))
    cam = small_camera((40, 44), 2.0)
    poses = synth.sample_poses(vol, synth.gt_pose(vol), 4, 25.0, 5.0, seed=2)
    rc = xr.RayCasterLineIntCUDA()
    rc.set_camera_model(cam)
    rc.set_ray_step_size(0.25)
    rc.set_num_projs(len(poses))
    rc.allocate_resources()
    rc.distribute_xforms_among_cam_models(poses)
    imgs, d_vox = [], _device(v)
    for device in (False, True):
        if device:
            rc.set_volumes_device([vol], [d_vox.data_ptr()], vt)
        else:
            rc.set_volume(vol, vt)
        for skip in (True, False):
            rc.set_empty_space_skipping(skip)
            for layout in (-1, 0):
                rc.set_launch_config(layout, 1, 4, 8)
                rc.compute()
                imgs.append(rc.projs())
    for img in imgs[1:]:
        np.testing.assert_array_equal(img, imgs[0])
    ref = oracle.drr_f32(v, oracle_geom(vol), oracle_cams([cam]), poses, step=0.25)
    rel, zero = drr_rel_err(imgs[0], ref)
    assert zero == 0.0 and rel <= tol, rel


@pytest.mark.parametrize("vt", [0, 1])
def test_one_volume_over_another(xr, vt):
    """A caster set to one volume after another renders what a new caster does,
    whichever sizes follow each other, and keeps its volume when one is refused."""
    cam = small_camera((40, 44), 3.0)
    rng = np.random.default_rng(3)

    def caster():
        rc = xr.RayCasterLineIntCUDA()
        rc.set_camera_model(cam)
        rc.set_ray_step_size(0.5)
        rc.set_num_projs(1)
        rc.allocate_resources()
        return rc

    def image(rc, vol):
        rc.distribute_xforms_among_cam_models(synth.gt_pose(vol)[None])
        rc.compute()
        return rc.projs()

    rc = caster()
    for size in ((40, 36, 44), (40, 36, 44), (36, 40, 30), (64, 60, 50), (8, 9, 10), (64, 60, 50)):
        vol = api.Volume(rng.uniform(0.0, 1.0, size[::-1]).astype(np.float32))
        new, d_vox = caster(), _device(vol.voxels)
        rc.set_volumes_device([vol], [d_vox.data_ptr()], vt)
        new.set_volume(vol, vt)
        want = image(new, vol)
        np.testing.assert_array_equal(image(rc, vol), want)
    if vt == 1:
        bad = vol.voxels.copy()
        bad[3, 4, 5] = np.inf
        with pytest.raises(XRegError):
            rc.set_volume(api.Volume(bad), 1)
        np.testing.assert_array_equal(image(rc, vol), want)
