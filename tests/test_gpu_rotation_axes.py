"""Rotations about one volume axis (shears of one coefficient, k_shear1, on a
work volume with the rotation axis fastest), about two, and tilt series that
share launches, against the FP64 oracle: relative L2 <= 1e-4 as in
test_rotation.py (the shears' FP32 transforms agree with 64 bits to about
1e-6)."""
import numpy as np
import pytest

from mset_b200 import Session
from oracle import oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("angles", [(25, 0, 0), (0, -40, 0), (0, 0, 33), (0, 11, 0), (90, 0, 0), (20, 15, 0),
                                    (0.2, 30, 0.1)], ids=str)
@pytest.mark.parametrize("n", [24, 32, 48, 64, 96])
def test_axis_rotation_matches_oracle(gpu_available, n, angles, inverse):
    v = np.random.default_rng(n).random((n, n, n)).astype(np.float32)
    ref = O.rot3d(v, angles, inverse=inverse)
    with Session() as s:
        out = s.rotate_volume(v, angles, inverse=inverse)
    assert rel_l2(out, ref) < 1e-4


@pytest.mark.parametrize("angles", [(0, -17, 0), (14, 0, 0), (0, 0, 40)], ids=str)
@pytest.mark.parametrize("n", [128, 160])
def test_axis_rotation_of_large_planes(gpu_available, n, angles):
    """against the line kernels, which turn volumes of any sides by other
    transforms (1e-5, as in test_gpu_line_rotation_of_a_cubic_volume_equals_plane_rotation)"""
    v = np.random.default_rng(n).random((n, n, n)).astype(np.float32)
    with Session() as s:
        planes = s.rotate_volume(v, angles)
        lines = s.rotate_volume(v, angles, lines=True)
    assert rel_l2(planes, lines) < 1e-5


@pytest.mark.parametrize("axes", ["y", "yz", "x"])
@pytest.mark.parametrize("n,window", [(24, 32), (32, 32)])
def test_rotations_in_shared_launches_match_oracle(gpu_available, n, window, axes):
    """the update of one iteration over 18 tilts (two launch groups), one of
    them unturned, about one axis or about two.  The step is taken from the
    oracle's own gradient so that the largest update is 5% of the largest voxel:
    FP32 storage then resolves the update to 2^-24 / 0.05 = 1e-6 of its largest
    value, and the FP32 gradients agree with 64 bits to about 1e-5"""
    from mset_b200.batch import BatchSession
    from tests.helpers import small_case
    from tests.iteration_oracle import iterate

    c = small_case(n=window, nz=n, npos=2, b=2, seed=5, defocus=15.0, jitter=3.0, strength=20.0)
    J = 18
    ang = np.zeros((J, 3), np.float32)
    th = np.linspace(-40, 44, J).round(2)
    th[7] = 0.0
    ang[:, {"y": 1, "yz": 1, "x": 2}[axes]] = th
    if axes == "yz":
        ang[9:, 1], ang[9:, 0] = 0.0, th[9:]
    rec = (np.random.default_rng(3).random((n, n, n)) * 20).astype(np.float32)

    def oracle(step):
        tilts = [dict(probe=c["probe"], sx=c["sx"], sy=c["sy"], meas=c["meas"]) for _ in range(J)]
        return iterate(rec.astype(np.float64), tilts, c["prop"], [a.astype(float) for a in ang], sigma=c["sigma"],
                       dz=c["dz"], binning=2, step=(step, 0.0, 0.0), positivity=False)

    unit, errs = oracle(1.0)
    step = float(np.float32(0.05 * rec.max() / np.abs(unit - rec).max()))
    ref = rec + step * (unit - rec)
    bs = BatchSession(n=window, nz=n, npos=[2] * J, prop=c["prop"], sigma=c["sigma"], potential_pixelsize=c["dz"],
                      slice_binning=2, step_size=(step, 0.0, 0.0))
    for j in range(J):
        bs.set_tilt(j, probe=c["probe"], scan_x=c["sx"], scan_y=c["sy"], measured=c["meas"])
    bs.iteration_setup(n, ang, positivity=False)
    bs.set_rec(rec)
    err, _ = bs.iterate(1)
    out = bs.get_rec()
    bs.close()
    assert rel_l2(out - rec, ref - rec) < 1e-4
    assert rel_l2(err[0], errs) < 1e-4
