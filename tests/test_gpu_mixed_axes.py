"""Tilts about x, y and z in one launch group: every work volume keeps its own
fastest axis, and the gradient sum goes over runs of tilts that share a tile
axis, in order.  Against the FP64 oracle (relative L2 <= 1e-4, the step taken so
that FP32 storage resolves the update: see
test_rotations_in_shared_launches_match_oracle)."""
import numpy as np
import pytest

from mset_b200.batch import BatchSession
from tests.helpers import rel_l2, small_case
from tests.iteration_oracle import iterate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [(2, 1, 0), (0, 1, 2, 1), (1, 1, 0, 0, 2)], ids=str)
@pytest.mark.parametrize("n,window", [(24, 32), (32, 32)])
def test_tilts_about_three_axes_match_oracle(gpu_available, n, window, columns):
    c = small_case(n=window, nz=n, npos=2, b=2, seed=9, defocus=15.0, jitter=3.0, strength=20.0)
    J = 7
    ang = np.zeros((J, 3), np.float32)
    for j, th in enumerate((-35, -21, 0, 14, 18, 29, 42)):
        ang[j, columns[j % len(columns)]] = th
    rec = (np.random.default_rng(4).random((n, n, n)) * 20).astype(np.float32)
    tilts = [dict(probe=c["probe"], sx=c["sx"], sy=c["sy"], meas=c["meas"]) for _ in range(J)]
    unit, errs = iterate(rec.astype(np.float64), tilts, c["prop"], [a.astype(float) for a in ang], sigma=c["sigma"],
                         dz=c["dz"], binning=2, step=(1.0, 0.0, 0.0), positivity=False)
    step = float(np.float32(0.05 * rec.max() / np.abs(unit - rec).max()))
    bs = BatchSession(n=window, nz=n, npos=[2] * J, prop=c["prop"], sigma=c["sigma"], potential_pixelsize=c["dz"],
                      slice_binning=2, step_size=(step, 0.0, 0.0))
    for j in range(J):
        bs.set_tilt(j, probe=c["probe"], scan_x=c["sx"], scan_y=c["sy"], measured=c["meas"])
    bs.iteration_setup(n, ang, positivity=False)
    bs.set_rec(rec)
    err, _ = bs.iterate(1)
    out = bs.get_rec()
    bs.close()
    assert rel_l2(out - rec, step * (unit - rec)) < 1e-4
    assert rel_l2(err[0], errs) < 1e-4
