"""The sequential modes on a cluster per field (seq_kernel.cuh) against the
same pass on the one-CTA shapes (mset_set_sequential_split(0)), at every window
and where the kernel's paths differ: a last slab of fewer planes, more planes
than it fetches ahead, one slab, one position, the exact adjoint, a propagator
that is no product of two vectors.

Both run the same FP32 operations per element in the same order; only the FP64
sums' order may differ, so the changes agree to 1e-5 as in
test_sequential_pass_on_a_cluster_equals_one_cta.  24^2 and 32^2 run on one
CTA either way and are compared with the FP64 oracle (1e-4)."""
import numpy as np
import pytest

from mset_b200 import MSET_ADJOINT_EXACT, MSET_ADJOINT_REF, MSET_MODE_MSET, MSET_MODE_SSET, Session
from oracle import oracle as O
from tests.helpers import reasonable_steps, rel_l2, small_case
from tests.test_gpu_parity import STRENGTH, TOL, coord_tol

pytestmark = pytest.mark.gpu

OPTIONS = [  # method, adjoint, nz, binning, positions, separable propagator
    (MSET_MODE_MSET, MSET_ADJOINT_REF, 7, 3, 3, True),
    (MSET_MODE_MSET, MSET_ADJOINT_EXACT, 5, 2, 2, False),
    (MSET_MODE_MSET, MSET_ADJOINT_REF, 1, 1, 1, True),
    (MSET_MODE_SSET, MSET_ADJOINT_EXACT, 4, 1, 2, True),
]


def _run(c, step, method, adjoint, split):
    with Session() as s:
        s.set_sequential_split(split)
        s.upload(c["V"], c["probe"], c["prop"], sigma=c["sigma"], potential_pixelsize=c["dz"], scan_x=c["sx"],
                 scan_y=c["sy"], measured=c["meas"], step_size=step, slice_binning=c["b"])
        return s.run(method, adjoint)


@pytest.mark.parametrize("option", OPTIONS, ids=["ref-z7b3", "exact-fullprop", "one-slab", "sset-exact"])
@pytest.mark.parametrize("n", [24, 32, 48, 64, 96, 128, 160, 256])
def test_cluster_pass_equals_one_cta_pass(gpu_available, n, option):
    method, adjoint, nz, b, npos, sep = option
    c = small_case(n=n, nz=nz, npos=npos, b=b, seed=n + nz, defocus=20.0, jitter=4.0, strength=STRENGTH)
    if not sep:
        k = np.linspace(-1, 1, n)
        c["prop"] = (c["prop"] * np.exp(0.3j * np.outer(k, k))).astype(np.complex64)
    step = reasonable_steps(c, method, adjoint)
    rv1, pr1, sx1, sy1, e1 = _run(c, step, method, adjoint, True)
    one_cta = n <= 32
    if one_cta:
        rv0, pr0, sx0, sy0, e0 = O.run_tilt(c["V"], c["probe"], c["prop"], c["sx"], c["sy"], c["meas"],
                                            sigma=c["sigma"], dz=c["dz"], step=step, binning=b, method=method,
                                            adjoint=adjoint)
        e0 = e0 / npos / n ** 2
    else:
        rv0, pr0, sx0, sy0, e0 = _run(c, step, method, adjoint, False)
    tol = TOL if one_cta else 1e-5
    assert rel_l2(rv1 - c["V"], rv0 - c["V"]) < tol
    assert rel_l2(pr1 - c["probe"], pr0 - c["probe"]) < tol
    d0 = np.r_[sx0 - c["sx"], sy0 - c["sy"]]
    assert rel_l2(np.r_[sx1 - c["sx"], sy1 - c["sy"]], d0) < coord_tol(n, np.r_[c["sx"], c["sy"]], d0)
    assert abs(e1 - e0) <= tol * e0
