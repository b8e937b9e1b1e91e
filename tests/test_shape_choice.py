"""Which compiled shape a batched session runs on, by its positions per SM
(csrc/mset_dispatch.cu, kAllGeos): the names of the kernels its pass launches, on
a CUDA runtime of host memory with 148 SMs (hostcuda.py)."""
import re

import pytest

from tests import hostcuda

# window, positions per SM -> threads and CTAs per SM that the shape is compiled for
CASES = [(24, 1, (192, 4)), (24, 20, (192, 4)), (32, 1, (128, 4)), (48, 2, (192, 2)), (48, 3, (192, 4)),
         (64, 6, (256, 2)), (64, 7, (128, 4)), (96, 1, (384, 1)), (96, 2, (384, 2)), (160, 1, (640, 1)),
         (160, 3, (640, 1))]


@pytest.mark.parametrize("n,per_sm,shape", CASES)
def test_shape_by_positions_per_sm(n, per_sm, shape):
    r = hostcuda.run(f"""
b = batched({n}, [148 * {per_sm}], nz=2)
F.fake_clear_log()
b.gradient(want=("err",))
b.close()
report(names=launched())
""")
    names = [x for x in r["names"] if "k_positions" in x]
    assert len(names) == 1
    got = re.search(r"3GeoILi(\d+)ELi(\d+)ELi(\d+)ELi(\d+)E", names[0])
    assert got and int(got[1]) == n and (int(got[3]), int(got[4])) == shape, names


def test_the_repeated_positions_of_the_shape_test_reach_another_shape():
    """test_gpu_shapes.py compares a session of 4 positions with one of 3, 7 and
    2 positions per SM at 48, 64 and 96: those are different kernels"""
    r = hostcuda.run("""
got = {}
for n, per_sm in ((48, 3), (64, 7), (96, 2)):
    for npos in (4, per_sm * 148 // 4 * 4):
        b = batched(n, [npos], nz=2)
        F.fake_clear_log()
        b.gradient(want=("err",))
        b.close()
        got.setdefault(n, []).append([x for x in launched() if "k_positions" in x])
report(got=got)
""")
    for n, (small, many) in r["got"].items():
        assert len(small) == len(many) == 1 and small != many, n
