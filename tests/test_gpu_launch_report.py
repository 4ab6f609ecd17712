"""The launch configuration that is reported after an evaluation is the one that ran:
job steps always trim rays to their occupied macro cells (loop 3 or above) in blocks of
at most 4 warps across; fused ones have 8."""
import numpy as np
import pytest

from tests.helpers import small_camera, small_volume
from xreg_gb300 import synth

pytestmark = pytest.mark.gpu


def _objective(xr, vt, bw, loop):
    vol, cam = small_volume(9, (40, 36, 44), (1.5, 1.5, 1.5)), small_camera((36, 40), 3.0)
    rc = xr.RayCasterLineIntCUDA()
    rc.set_volume(vol, vt)
    rc.set_camera_model(cam)
    rc.set_launch_config(2 if vt == 0 else 1, bw, loop, 4)
    m = xr.ImgSimMetric2DGradNCCCUDA()
    m.set_fixed_image(np.random.default_rng(2).random((36, 40)).astype(np.float32))
    poses = synth.sample_poses(vol, synth.gt_pose(vol), 3, 10.0, 10.0, seed=6)
    return rc, m, xr.PopulationObjective(rc, [m], 3), poses


@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("bw,loop", [(2, 1), (2, 2), (4, 3), (8, 4), (1, 6)])
def test_job_steps(xr, vt, bw, loop):
    layout, values = (2 if vt == 0 else 1), []
    for fused in (False, True):
        rc, m, obj, poses = _objective(xr, vt, bw, loop)
        js = xr.JobSet()
        js.set_fused(fused)
        values.append(js.eval([obj], [poses])[0])
        assert rc.launch_config_ex() == (layout, bw if fused else min(bw, 4), max(loop, 3), 4)
    rc, m, obj, poses = _objective(xr, vt, bw, loop)
    values.append(obj.eval(poses))
    assert rc.launch_config_ex() == (layout, bw, loop, 4)
    np.testing.assert_array_equal(values[0], values[1])
    np.testing.assert_array_equal(values[0], values[2])
