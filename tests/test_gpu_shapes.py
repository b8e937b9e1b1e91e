"""The batched kernel's shapes and the orders of its per-slab fields: every
window against the FP64 oracle (1e-4, as in test_gpu_parity.py) with the adjoint,
method and checkpoint options that read the saved waves differently, and the
shapes chosen by positions per SM against the small session's shape.  (The
scan-position sums of these inputs cancel to a few 1e-4 in FP32 whatever the
shape; the second test compares them between shapes.)

In the second test every session sees the same few positions, repeated: the
gradient sums are the small session's times the repetitions.  The shapes run
the same FP32 operations, so 1e-6 covers the FP64 sums and the compiler's
choice of fused operations at a few places."""
import numpy as np
import pytest
import torch

from mset_b200 import MSET_ADJOINT_EXACT, MSET_ADJOINT_REF, MSET_MODE_MSET, MSET_MODE_SSET
from mset_b200.batch import BatchSession
from oracle import oracle as O
from tests.helpers import rel_l2, small_case
from tests.test_gpu_parity import STRENGTH, TOL

pytestmark = pytest.mark.gpu


def _session(c, npos, *, method=MSET_MODE_MSET, adjoint=MSET_ADJOINT_REF, reps=1, ckpt=0):
    bs = BatchSession(n=c["V"].shape[1], nz=c["V"].shape[0], npos=[npos * reps], prop=c["prop"], sigma=c["sigma"],
                      potential_pixelsize=c["dz"], slice_binning=c["b"], method=method, adjoint=adjoint)
    bs.set_tilt(0, probe=c["probe"], scan_x=np.tile(c["sx"], reps), scan_y=np.tile(c["sy"], reps),
                measured=np.tile(c["meas"], (reps, 1, 1)), volume=c["V"])
    bs.set_checkpoint(ckpt)
    return bs


@pytest.mark.parametrize("method,adjoint,ckpt", [(MSET_MODE_MSET, MSET_ADJOINT_REF, 0),
                                                 (MSET_MODE_MSET, MSET_ADJOINT_EXACT, 2),
                                                 (MSET_MODE_MSET, MSET_ADJOINT_REF, 3),
                                                 (MSET_MODE_SSET, MSET_ADJOINT_EXACT, 0)],
                         ids=["ref", "exact-ck2", "ref-ck3", "sset-exact"])
@pytest.mark.parametrize("n", [24, 32, 48, 64, 96, 128])
def test_window_matches_oracle(gpu_available, n, method, adjoint, ckpt):
    c = small_case(n=n, nz=7, npos=3, b=2 if ckpt != 3 else 1, seed=50 + n, defocus=15.0, jitter=3.0,
                   strength=STRENGTH)
    bs = _session(c, 3, method=method, adjoint=adjoint, ckpt=ckpt)
    out = bs.gradient()
    err = bs.error()
    inten = bs.simulate()
    bs.close()
    g, pa, pd, e = O.batched_tilt(c["V"], c["probe"], c["prop"], c["sx"], c["sy"], c["meas"], sigma=c["sigma"],
                                  dz=c["dz"], binning=c["b"], method=method, adjoint=adjoint)
    assert rel_l2(out["grad"][0], g) < TOL
    assert rel_l2(np.fft.fft2(out["probe"][0]), pa) < TOL
    assert abs(out["err"][0] - e) <= TOL * e and abs(err[0] - e) <= TOL * e
    o = O.position(c["V"], c["probe"], c["prop"], c["sx"][1], c["sy"][1], O.amp_std(c["meas"][1]), sigma=c["sigma"],
                   dz=c["dz"], binning=c["b"], method=method)
    assert rel_l2(inten[1], np.fft.fftshift(np.abs(o["far"]) ** 2)) < TOL


@pytest.mark.parametrize("n,per_sm", [(48, 3), (64, 7), (96, 2)])
def test_shape_for_many_positions_equals_small_session(gpu_available, n, per_sm):
    npos = 4
    c = small_case(n=n, nz=3, npos=npos, b=1, seed=60 + n, defocus=15.0, jitter=3.0, strength=STRENGTH)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    reps = per_sm * sms // npos
    small, many = _session(c, npos), _session(c, npos, reps=reps)
    a, b = small.gradient(), many.gradient()
    shape_a, shape_b = small.shape(), many.shape()
    small.close()
    many.close()
    assert shape_a["threads"] > 0 and shape_b["threads"] > 0
    assert rel_l2(b["grad"] / reps, a["grad"]) < 1e-6
    assert rel_l2(b["probe"] / reps, a["probe"]) < 1e-6
    assert rel_l2(b["posdir"][:npos], a["posdir"]) < 1e-6
    assert abs(b["err"][0] / reps - a["err"][0]) <= 1e-6 * a["err"][0]
