"""The unclamped reads of the cell copy, restated on the host from the kernel's own
headers (xr_xfloat.h, xr_cells.h): for ordinary views every sample of every ray
reads the cell of its position, and for frames that hold NaN, infinities or numbers
that float cannot carry no ray is left to the unclamped march, whose address would
lie outside the copy."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from xreg_gb300 import synth
from xreg_gb300.api import CameraModel
from xreg_gb300.se3 import euler_xyz, rigid

ROOT = Path(__file__).resolve().parents[1]
F32, F16, BF16 = 0, 1, 2


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = tmp_path_factory.mktemp("cells") / "ray_cells_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-frounding-math", "-ffp-contract=off", f"-I{ROOT / 'xreg_gb300' / 'csrc'}",
                    f"-I{ROOT / 'include'}", str(ROOT / "tests/cpp/ray_cells_check.cpp"), "-o", str(out)], check=True)
    return out


def _volume(size):
    return synth.phantom_volume(size, (1.5, 1.25, 1.75), 3)


def _camera(rows=21, cols=19, px=9.0):
    return CameraModel.naive(synth.SDD_MM, rows, cols, px, px)


def _views(vol):
    gt = synth.gt_pose(vol)
    C = vol.xform_img_center_to_itk_phys()
    turned = [C @ rigid(euler_xyz(*np.radians(a)), np.zeros(3)) @ np.linalg.inv(C) @ gt
              for a in ((0.0, 0.0, 0.0), (90.0, 0.0, 0.0), (0.0, 90.0, 0.0), (30.0, 50.0, 10.0))]
    return list(synth.sample_poses(vol, gt, 4, 20.0, 10.0, seed=5)) + turned


def _run(exe, tmp_path, vol, cam, poses, vt=F32, step=0.5, guard=True, intrins=None):
    p2i = np.linalg.inv(vol.index_to_phys())
    K = cam.intrins if intrins is None else intrins
    rows = []
    for p in poses:
        rows.append(np.concatenate([np.array(vol.size, float), [vt, step, cam.num_det_rows, cam.num_det_cols, guard],
                                    np.asarray(K, float).ravel(), np.asarray(cam.extrins, float).ravel(),
                                    [cam.focal_len, cam.desc.coord_frame_type], p2i[:3, :3].ravel(), p2i[:3, 3], p[:3, :3].ravel(), p[:3, 3]]))
    fi, fo = tmp_path / "in.f64", tmp_path / "out.f64"
    with np.errstate(invalid="ignore", over="ignore"):
        np.concatenate(rows).astype(np.float64).tofile(fi)
    subprocess.run([str(exe), str(fi), str(fo)], check=True)
    out = np.fromfile(fo).reshape(len(poses), 6)
    return dict(zip(("hits", "unclamped", "samples", "outside", "wrong", "guarded"), out.T))


@pytest.mark.parametrize("vt", [F32, F16, BF16])
@pytest.mark.parametrize("size", [(31, 5, 30), (31, 40, 31), (40, 36, 44), (200, 17, 9), (65, 130, 21)])
def test_ordinary_views_read_the_cell_of_every_sample(exe, tmp_path, size, vt):
    vol = _volume(size)
    c = _run(exe, tmp_path, vol, _camera(), _views(vol), vt)
    assert c["samples"].sum() > 1000
    assert np.all(c["unclamped"] == c["hits"]) and np.all(c["guarded"] == 0)
    assert np.all(c["outside"] == 0) and np.all(c["wrong"] == 0)


def _broken(vol):
    """Poses that a device buffer may hold, or whose doubles float cannot carry."""
    gt = synth.gt_pose(vol)
    out = []
    for value in (np.nan, np.inf, -np.inf, 1e39, -1e300, 3e38, 1e30, 1e20):
        for where in ((0, 0), (2, 1), (0, 3), (2, 3), (slice(0, 3), slice(0, 3)), (slice(0, 3), 3), (slice(0, 3), slice(0, 4))):
            p = gt.copy()
            p[where] = value
            out.append(p)
    return out


@pytest.mark.parametrize("vt", [F32, F16, BF16])
def test_no_read_outside_the_copy_for_frames_that_are_not_finite(exe, tmp_path, vt):
    vol, cam = _volume((40, 36, 44)), _camera()
    c = _run(exe, tmp_path, vol, cam, _broken(vol), vt)
    assert np.all(c["outside"] == 0) and np.all(c["wrong"] == 0)
    # and the guard is what keeps them: without it such rays would read elsewhere
    free = _run(exe, tmp_path, vol, cam, _broken(vol), vt, guard=False)
    assert np.all(free["hits"] == c["hits"]) and free["outside"].sum() > 0
    assert c["guarded"].sum() > 0
    for intrins in (np.zeros((3, 3)), np.full((3, 3), np.nan), np.full((3, 3), np.inf)):  # no ray at all, or none unclamped
        c = _run(exe, tmp_path, vol, cam, _views(vol) + _broken(vol), vt, intrins=intrins)
        assert np.all(c["outside"] == 0) and np.all(c["wrong"] == 0)


@pytest.mark.parametrize("vt", [F32, F16, BF16])
def test_focal_points_far_away(exe, tmp_path, vt):
    """A focal point so far away that the start of a ray rounds by voxels."""
    vol = _volume((40, 36, 44))
    seen = 0
    for far in (1e4, 1e6, 1e7, 1e8, 1e9):
        cam = CameraModel.naive(far, 21, 19, 9.0, 9.0)
        C = vol.xform_img_center_to_itk_phys()
        view = np.array([[1.0, 0, 0], [0, 0, 1.0], [0, -1.0, 0]])
        poses = [C @ rigid(np.eye(3), d) @ rigid(view, view @ np.array([0.0, 0.0, far - 100.0])) for d in np.array([[0, 0, 0], [3.3, 7.7, 1.1], [9.0, 2.0, 5.0]])]
        c = _run(exe, tmp_path, vol, cam, poses, vt)
        seen += c["hits"].sum()
        assert np.all(c["outside"] == 0)
        if far <= 1e6:
            assert np.all(c["guarded"] == 0)
    assert seen > 0


def _numbering(exe, n, vt):
    out = subprocess.run([str(exe), *map(str, n), str(vt), "numbering"], check=True, capture_output=True, text=True).stdout.split()
    return bool(int(out[0])), (int(out[1]), int(out[2])), int(out[3]), int(out[4]), tuple(map(float, out[5:]))


# full volumes, stacks of few slices on each axis, axes as long as 2^31 voxels allow
@pytest.mark.parametrize("n", [(256, 256, 256), (512, 512, 300), (1290, 1290, 1290), (512, 512, 4), (4, 512, 512), (512, 4, 512),
                               (2, 2, 2), (55, 9, 55), (56, 9, 54), (20000, 20000, 4), (32768, 32767, 2), (2, 32768, 32767),
                               (4194303, 2, 2), (2, 4194303, 2), (2, 2, 4194303), (440000000, 2, 2), (2, 440000000, 2),
                               (2, 2, 440000000), (536870911, 2, 2), (2, 536870911, 2), (2, 2, 536870911), (4194303, 255, 2)])
@pytest.mark.parametrize("vt", [F32, F16, BF16])
def test_cell_numbers_fit_their_32_bits(exe, n, vt):
    numbered, (sx, sy), nbytes, in_bytes, kfl = _numbering(exe, n, vt)
    cell = 32 if vt == F32 else 16
    least = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    if not numbered:
        assert least >= 2 ** 32 and (sx, sy, nbytes) == (0, 0, 0) and kfl == (0.0, 0.0, 0.0)
        return
    assert sx >= n[2] + 1 and sy >= sx * (n[0] + 1) and nbytes == sy * (n[1] + 1) * cell < 2 ** 32 * cell
    assert nbytes <= 1.27 * least * cell  # an eighth on either stride
    assert in_bytes == (nbytes < 2 ** 32)
    if kfl != (0.0, 0.0, 0.0):
        unit, s = (cell if in_bytes else 1), (32768.0 if vt == F16 else 1.0)
        for k in range(3):
            one = s if k < 2 else 1.0
            m = kfl[k] / one - 2.0 ** 23
            assert m == int(m) and 1 <= m and m + n[k] < 2 ** 23  # 2^23 + m + floor(p) stays below 2^24
        b = [0x52800000 if vt == F16 else 0x4B000000] * 2 + [0x4B000000]
        at = [b[k] + int(kfl[k] / (s if k < 2 else 1.0) - 2.0 ** 23) for k in range(3)]  # of position 0: cell 1
        got = (at[1] * sy * unit + at[0] * sx * unit + at[2] * unit) % 2 ** 32
        assert got == (sy + sx + 1) * unit % 2 ** 32


@pytest.mark.parametrize("n", [(512, 512, 300), (256, 256, 256), (512, 512, 4), (4, 512, 512), (33, 40, 55), (20000, 20000, 4),
                               (440000000, 2, 2), (2, 2, 536870911)])
@pytest.mark.parametrize("vt", [F32, F16, BF16])
def test_the_servers_budget_counts_the_copy(exe, n, vt):
    from types import SimpleNamespace

    from xreg_gb300.regi import Registration, RegiLevel, cell_copy_bytes
    numbered, _, nbytes, _, _ = _numbering(exe, n, vt)
    assert cell_copy_bytes(n, vt) == nbytes
    job = Registration.__new__(Registration)
    job.vol, job.voxel_type = SimpleNamespace(size=n), vt
    job.levels = [RegiLevel([_camera()], [np.zeros((21, 19), np.float32)])]
    assert job.footprint_bytes() >= n[0] * n[1] * n[2] * (4 if vt == F32 else 2) + nbytes
