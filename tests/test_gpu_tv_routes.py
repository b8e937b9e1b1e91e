"""The TV routes where the choice between them changes (csrc/mset_volume.cu,
tv_cluster_pays): volumes of few and of many slices per CTA, thin ones, and rows
that are no whole float4 groups, against the numpy restatement (oracle/tv.py)
within the bound derived in test_gpu_tv_kernels.py."""
import numpy as np
import pytest

from mset_b200 import Session
from oracle import tv
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [  # (n3, n2, n1)
    (48, 24, 24), (64, 24, 24), (64, 16, 16), (100, 4, 4),           # either side of the cluster's end
    (80, 32, 32), (8, 48, 48), (400, 16, 16), (3, 40, 40),           # marching
    (32, 33, 31), (9, 50, 50), (200, 9, 9), (34, 34, 34),            # cluster, several columns or many slices
    (500, 6, 6), (1000, 5, 5),                                       # two kernels
]


@pytest.mark.parametrize("fista", [True, False], ids=["fista", "tv"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_tv_route_matches_oracle(gpu_available, shape, fista):
    v = np.random.default_rng(sum(shape)).random(shape).astype(np.float32)
    with Session() as s:
        for niter in (1, 40, 7):
            ref, _ = tv.tv_method(v, 0.05, niter, fista=fista)
            assert rel_l2(s.tv(v, 0.05, niter, fista), ref) < 1e-5, niter
