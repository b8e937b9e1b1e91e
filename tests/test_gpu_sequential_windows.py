"""The sequential modes at every window really run on the cluster they are
documented for, and agree with the one-CTA kernels where test_gpu_sequential.py
and test_gpu_steps.py do not look: the reference's adjoint of single-slice tilts,
passes of more positions, and the per-position steps at 48^2 (odd transforms),
96^2 and 160^2 (16 CTAs).

Both run the same FP32 operations per element, only the FP64 sums' order may
differ: 1e-5, as in test_gpu_sequential.py.  (The steps' scan-position sums
against 64 bits are limited by FP32 cancellation at 96^2 and 160^2 whatever the
kernel, so the steps are compared with the one-CTA kernel.)"""
import numpy as np
import pytest

from mset_b200 import MSET_ADJOINT_EXACT, MSET_ADJOINT_REF, MSET_MODE_MSET, MSET_MODE_SSET, Session
from tests import test_gpu_sequential as sequential
from tests import test_gpu_steps as steps
from tests.helpers import reasonable_steps, rel_l2, small_case
from tests.test_gpu_parity import coord_tol

pytestmark = pytest.mark.gpu

CTAS = {24: 1, 32: 1, 48: 8, 64: 8, 96: 16, 128: 8, 160: 16, 256: 16}


@pytest.mark.parametrize("n", CTAS)
def test_ctas_per_field(gpu_available, n):
    c = small_case(n=n, nz=2, npos=1, seed=n)
    for split in (True, False):
        with Session() as s:
            s.set_sequential_split(split)
            s.upload(c["V"], c["probe"], c["prop"], sigma=c["sigma"], potential_pixelsize=c["dz"], scan_x=c["sx"],
                     scan_y=c["sy"], measured=c["meas"], step_size=(0.0, 0.0, 0.0))
            assert s.sequential_split() == (CTAS[n] if split else 1)


@pytest.mark.parametrize("option", [(MSET_MODE_SSET, MSET_ADJOINT_REF, 4, 1, 3, True),
                                    (MSET_MODE_MSET, MSET_ADJOINT_REF, 4, 1, 12, True),
                                    (MSET_MODE_MSET, MSET_ADJOINT_EXACT, 3, 1, 12, True)],
                         ids=["sset-ref", "ref-12", "exact-12"])
@pytest.mark.parametrize("n", [n for n in CTAS if n > 32])
def test_cluster_pass_equals_one_cta_pass(gpu_available, n, option):
    sequential.test_cluster_pass_equals_one_cta_pass(gpu_available, n, option)


@pytest.mark.parametrize("n", [24, 32])
def test_small_windows_match_oracle(gpu_available, n):
    sequential.test_cluster_pass_equals_one_cta_pass(gpu_available, n, (MSET_MODE_SSET, MSET_ADJOINT_REF, 4, 1, 3, True))


@pytest.mark.parametrize("method,admode", steps.MODES + [(MSET_MODE_SSET, MSET_ADJOINT_EXACT)],
                         ids=["mset-ref", "mset-exact", "sset-ref", "sset-exact"])
@pytest.mark.parametrize("case", [dict(n=48, nz=5, b=2), dict(n=96, nz=4, b=1), dict(n=160, nz=3, b=2)],
                         ids=lambda c: f"n{c['n']}z{c['nz']}b{c['b']}")
def test_steps_equal_one_cta_steps(gpu_available, case, method, admode):
    n, k = case["n"], 1
    c = steps._case(case["n"], case["nz"], case["b"])
    step = reasonable_steps(c, method, admode)
    row, col = float(c["sx"][k]), float(c["sy"][k])
    got = []
    for split in (True, False):
        with Session() as s:
            s.set_sequential_split(split)
            steps._upload(s, c, step, 3)
            f = s.step02(k, row, col, mode=method)
            got.append((f, s.step03(mode=method, adjoint=admode)))
    (f1, g1), (f0, g0) = got
    for key in ("calc", "resi", "psi0", "waves"):
        assert rel_l2(f1[key], f0[key]) < 1e-5, key
    assert abs(f1["err"] - f0["err"]) <= 1e-5 * f0["err"]
    assert rel_l2(g1["grad"], g0["grad"]) < 1e-5
    assert rel_l2(g1["probe"] - c["probe"], g0["probe"] - c["probe"]) < 1e-5
    d0 = np.array([g0["row"] - row, g0["col"] - col])
    assert rel_l2(np.array([g1["row"] - row, g1["col"] - col]), d0) < coord_tol(n, [row, col], d0)
