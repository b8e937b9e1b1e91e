"""A session that iterates and is asked for rotations and TV of other sizes in
between gives what one that only iterates gives: work buffers and the twiddle
table are shared between these calls.  (Runs of one session differ by the order
of the FP64 sums, far below the FP32 state's 1e-6.)"""
import ctypes as C

import numpy as np
import pytest

from mset_b200._lib import check, fptr
from mset_b200.batch import BatchSession
from tests.helpers import rel_l2, small_case

pytestmark = pytest.mark.gpu

EYE = [np.eye(3, dtype=np.float32)[i].copy() for i in range(3)]


def _rotate(b, n):
    v = np.random.default_rng(n).random((n, n, n)).astype(np.float32)
    out = np.empty_like(v)
    check("mset_rotate_volume", b._lib.mset_rotate_volume(b._h, fptr(v), fptr(out), n, *[fptr(e) for e in EYE], 0.0, 20.0,
                                                          5.0, 0))


def _tv(b, *shape):
    v = np.random.default_rng(shape[0]).random(shape).astype(np.float32)
    check("mset_tv", b._lib.mset_tv(b._h, fptr(v), shape[2], shape[1], shape[0], 0.05, 3, 1, C.POINTER(C.c_double)()))


BETWEEN = {
    "nothing": lambda b: None,
    "smaller tv": lambda b: _tv(b, 24, 24, 24),
    "larger tv": lambda b: _tv(b, 64, 64, 64),
    "other rotations": lambda b: (_rotate(b, 24), _rotate(b, 96)),
    "all": lambda b: (_tv(b, 50, 50, 60), _rotate(b, 64), _tv(b, 8, 8, 8), _rotate(b, 32)),
}


def _iterated(between, graph, edge):
    c = small_case(n=48, nz=edge, npos=2, b=1, seed=3, defocus=15.0, jitter=3.0, strength=5.0)
    ang = np.array([[0, -20, 0], [0, 15, 3], [25, 0, 0]], np.float32)
    b = BatchSession(n=48, nz=edge, npos=[2] * 3, prop=c["prop"], sigma=c["sigma"], potential_pixelsize=c["dz"],
                     step_size=(1e-4, 1e-6, 1e-6))
    for j in range(3):
        b.set_tilt(j, probe=c["probe"], scan_x=c["sx"], scan_y=c["sy"], measured=c["meas"])
    b.iteration_setup(edge, ang, positivity=True, tv_lambda=1e-2, tv_iter=4)
    b.set_rec((np.random.default_rng(1).random((edge,) * 3) * 5).astype(np.float32))
    errs = []
    for _ in range(3):
        errs.append(b.iterate(1, graph)[0])
        between(b)
    out = b.get_rec()
    b.close()
    return out, np.array(errs)


@pytest.mark.parametrize("graph", [False, True], ids=["launches", "graph"])
@pytest.mark.parametrize("edge", [24, 48])
def test_iterations_with_other_calls_between_equal_iterations_alone(gpu_available, edge, graph):
    ref, errs = _iterated(BETWEEN["nothing"], graph, edge)
    for name in list(BETWEEN)[1:]:
        out, e = _iterated(BETWEEN[name], graph, edge)
        assert rel_l2(out, ref) < 1e-6, name
        assert rel_l2(e, errs) < 1e-6, name
