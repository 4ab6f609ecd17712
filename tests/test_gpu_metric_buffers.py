"""A metric that an objective uses: its values are read for as many images as the last
evaluation had, and when it is allocated again for fewer images with options that need
more room for each (a smaller stride, scores of every patch, another smoothing), a
population gets buffers of its size, alone and in a job set."""
import numpy as np
import pytest

from tests.helpers import small_camera, small_volume
from xreg_gb300 import synth

pytestmark = pytest.mark.gpu

SHAPE, POP = (60, 58), 300


def _metric(xr, kind):
    m = getattr(xr, kind)()
    m.set_fixed_image(np.random.default_rng(2).random(SHAPE).astype(np.float32))
    return m


def _options(m, smooth, stride, **options):
    if hasattr(m, "set_smooth_img_before_sobel_kernel_radius"):
        m.set_smooth_img_before_sobel_kernel_radius(smooth)
    if hasattr(m, "set_patch_stride"):
        m.set_patch_stride(stride)
        if options:
            m.set_patch_options(**options)


def _objective(xr, m):
    vol, cam = small_volume(9, (40, 36, 44), (1.5, 1.5, 1.5)), small_camera(SHAPE, 3.0)
    rc = xr.RayCasterLineIntCUDA()
    rc.set_volume(vol, 1)
    rc.set_camera_model(cam)
    return rc, xr.PopulationObjective(rc, [m], POP), synth.sample_poses(vol, synth.gt_pose(vol), POP, 10.0, 10.0, seed=6)


CASES = [("ImgSimMetric2DNCCCUDA", {}), ("ImgSimMetric2DGradNCCCUDA", {}), ("ImgSimMetric2DPatchNCCCUDA", {}),
         ("ImgSimMetric2DPatchNCCCUDA", {"save_all_per_patch_scores": 1}), ("ImgSimMetric2DPatchGradNCCCUDA", {}),
         ("ImgSimMetric2DPatchGradNCCCUDA", {"use_mov_img_patch_variances_as_wgts": 1}),
         ("ImgSimMetric2DPatchGradNCCCUDA", {"save_all_per_patch_scores": 1})]


@pytest.mark.parametrize("kind,options", CASES)
@pytest.mark.parametrize("smooth", [3, 5])
def test_metric_allocated_again_for_one_image(xr, kind, options, smooth):
    ref = _metric(xr, kind)
    _options(ref, smooth, 1, **options)
    _, obj0, poses = _objective(xr, ref)
    want = obj0.eval(poses)
    assert ref.num_moving_images() == POP
    np.testing.assert_array_equal(ref.sim_vals(), want)  # one view: the mean is its value

    m = _metric(xr, kind)
    _options(m, 0, 4)
    _, obj, _ = _objective(xr, m)
    obj.eval(poses[:3])
    _options(m, smooth, 1, **options)
    m.set_num_moving_images(1)
    m.allocate_resources()
    for n in (1, POP, POP, 5, POP):  # directly, and as captured
        np.testing.assert_array_equal(obj.eval(poses[:n]), want[:n])
        assert m.num_moving_images() == n
        np.testing.assert_array_equal(m.sim_vals(), want[:n])
    if options.get("save_all_per_patch_scores"):
        for i in (0, POP - 1):
            np.testing.assert_array_equal(m.patch_scores(i), ref.patch_scores(i))


@pytest.mark.parametrize("kind,options", [CASES[2], CASES[3]])
def test_in_a_job_set(xr, kind, options):
    ref = _metric(xr, kind)
    _options(ref, 5, 1, **options)
    _, obj0, poses = _objective(xr, ref)
    m = _metric(xr, kind)
    _options(m, 5, 4)
    _, obj, _ = _objective(xr, m)
    _options(m, 5, 1, **options)
    m.set_num_moving_images(1)
    m.allocate_resources()
    np.testing.assert_array_equal(xr.JobSet().eval([obj], [poses])[0], obj0.eval(poses))


def test_a_refused_step_binds_the_metric_to_its_population(xr):
    """A job step larger than the metric's allocation is refused, and allocating again
    then makes room for that step's population."""
    m = _metric(xr, "ImgSimMetric2DGradNCCCUDA")
    _, obj, poses = _objective(xr, m)
    want = obj.eval(poses[:40])
    m.set_num_moving_images(3)
    m.allocate_resources()
    js = xr.JobSet()
    with pytest.raises(xr.XRegError):
        js.eval([obj], [poses[:40]])
    assert m.num_moving_images() == 40
    m.allocate_resources()
    np.testing.assert_array_equal(js.eval([obj], [poses[:40]])[0], want)
