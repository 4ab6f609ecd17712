"""Volumes whose corner differences would not be finite (an infinite voxel, or one
above 2^126): they keep their cell copy, so that the layout asked for is the one
that runs, with the blend by weights; every layout gives the LINEAR layout's bits
and the oracle's finite pixels."""
import numpy as np
import pytest

from tests.helpers import drr_rel_err, oracle_cams, oracle_geom, small_camera
from xreg_gb300 import api, synth
from xreg_gb300.se3 import euler_xyz, rigid

pytestmark = pytest.mark.gpu

TOL = {0: 1e-4, 2: 2.0 ** -8}


def _poses(vol):
    gt = synth.gt_pose(vol)
    C = vol.xform_img_center_to_itk_phys()
    turned = [C @ rigid(euler_xyz(*np.radians(a)), np.zeros(3)) @ np.linalg.inv(C) @ gt
              for a in ((0.0, 0.0, 0.0), (90.0, 0.0, 0.0), (0.0, 90.0, 0.0))]
    return np.concatenate([synth.sample_poses(vol, gt, 2, 20.0, 5.0, seed=4), np.stack(turned)])


@pytest.mark.parametrize("vt", [0, 2])
@pytest.mark.parametrize("value", [np.inf, 2.0 ** 127])
@pytest.mark.parametrize("at", [(14, 20, 18), (0, 5, 39), (31, 34, 1), (32, 35, 39)])  # inside, on and beside faces
def test_cells_of_weighted_volumes(xr, oracle, vt, value, at):
    rng = np.random.default_rng(7)
    v = rng.uniform(0.5, 1.0, (33, 36, 40)).astype(np.float32)
    v[at] = value
    vol = api.Volume(v, spacing=(1.5, 1.5, 1.5))
    cam, poses = small_camera((45, 37), 4.0), _poses(vol)
    rc = xr.RayCasterLineIntCUDA()
    rc.set_volume(vol, vt)
    rc.set_camera_model(cam)
    rc.set_ray_step_size(0.5)
    rc.set_num_projs(len(poses))
    rc.allocate_resources()
    rc.distribute_xforms_among_cam_models(poses)
    rc.set_launch_config(0, 1, 4, 8)
    rc.compute()
    linear = rc.projs()
    for skip in (True, False):
        rc.set_empty_space_skipping(skip)
        for layout in ((1, 2, 3) if vt == 0 else (1,)):
            rc.set_launch_config(layout, 1, 4, 8)
            rc.compute()
            assert rc.launch_config_ex()[0] == layout
            np.testing.assert_array_equal(rc.projs(), linear)
        rc.set_launch_config(-1)
        rc.compute()
        assert rc.launch_config_ex()[0] == (2 if vt == 0 else 1)
        np.testing.assert_array_equal(rc.projs(), linear)
    ref = oracle.drr_f32(v, oracle_geom(vol), oracle_cams([cam]), poses, step=0.5)
    ok = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(linear), ok)
    rel, zero = drr_rel_err(np.where(ok, linear, 0.0), np.where(ok, ref, 0.0))
    assert zero == 0.0 and rel <= TOL[vt], rel


def test_job_sets_of_weighted_and_other_volumes(xr):
    """Job steps, fused and not, pose-grouped or not: every job's values and images are
    those of its objective alone."""
    rng = np.random.default_rng(11)
    cam, jobs = small_camera((45, 37), 4.0), []
    for vt, value in ((0, np.inf), (0, 1.0), (2, 2.0 ** 127), (2, 1.0), (1, 1.0), (0, 2.0 ** 127)):
        v = rng.uniform(0.5, 1.0, (33, 36, 40)).astype(np.float32)
        v[14, 20, 18] = value
        vol = api.Volume(v, spacing=(1.5, 1.5, 1.5))
        rc = xr.RayCasterLineIntCUDA()
        rc.set_volume(vol, vt)
        rc.set_camera_model(cam)
        rc.set_ray_step_size(0.5)
        m = xr.ImgSimMetric2DGradNCCCUDA()
        m.set_fixed_image(rng.random((45, 37)).astype(np.float32))
        jobs.append((rc, m, xr.PopulationObjective(rc, [m], 5), _poses(vol)))
    alone, images = [], []
    for rc, _, obj, poses in jobs:
        alone.append(obj.eval(poses))
        images.append(rc.projs())
    assert sum(np.isnan(i).any() or np.isinf(i).any() or i.max() > 1e30 for i in images) == 3
    for mode in ("split", "groups", "fused"):
        js = xr.JobSet()
        js.set_fused(mode == "fused")
        js.set_pose_groups(2 if mode == "groups" else 0)
        got = js.eval([j[2] for j in jobs], [j[3] for j in jobs])
        for (rc, _, _, _), g, a, i in zip(jobs, got, alone, images):
            np.testing.assert_array_equal(g, a)
            np.testing.assert_array_equal(rc.projs(), i)
