"""The TV kernels' routes against the numpy restatement (oracle/tv.py): all
iterations in one cluster launch, one marching kernel per iteration, and two
kernels where rows are no whole float4 groups; slices, rows and columns that do
not divide by the kernels' tiles, and the periodic edges of one-slice and
one-row volumes.

Tolerance: the dual field is FP32 with values of order 1; each of the (at most
40) projected steps adds rounding of a few 2^-24 and the projection does not
amplify it, so the output, input - lambda div(P) with lambda 0.05 and six terms
of P per voxel, is within 40 * 4 * 2^-24 * 6 * 0.05 = 3e-6 of inputs of order 1:
relative L2 < 1e-5."""
import numpy as np
import pytest

from mset_b200 import Session
from oracle import tv
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [  # (n3, n2, n1)
    (24, 24, 24), (32, 32, 32), (5, 7, 12), (9, 3, 17), (1, 16, 16), (30, 1, 8), (2, 2, 2),  # one cluster
    (21, 47, 96), (19, 33, 64), (40, 300, 4), (1, 130, 128), (17, 20, 260),                    # marching
    (40, 60, 50), (33, 64, 65),                                                                # two kernels
]


@pytest.mark.parametrize("fista", [True, False], ids=["fista", "tv"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_tv_route_matches_oracle(gpu_available, shape, fista):
    v = np.random.default_rng(sum(shape)).random(shape).astype(np.float32)
    for niter in (0, 1, 40, 7):  # an odd count ends in the other dual field
        ref, _ = tv.tv_method(v, 0.05, niter, fista=fista)
        with Session() as s:
            out = s.tv(v, 0.05, niter, fista)
            again = s.tv(v, 0.05, niter, fista)
        assert rel_l2(out, ref) < 1e-5, niter
        assert np.array_equal(out, again)
