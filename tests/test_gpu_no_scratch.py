"""The sequential pass and the per-position steps without memory for the cluster
kernels' scratch run on the one-CTA kernels at every window: the library in a
process whose device allocations of that size fail (deny_malloc.c), against the
same calls with the scratch (FP32 operations per element are the same ones, so
1e-5 as in test_gpu_sequential.py)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.helpers import reasonable_steps, rel_l2, small_case
from tests.test_gpu_parity import STRENGTH, coord_tol

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SCRIPT = """
import sys
import numpy as np
from mset_b200 import Session
d = np.load(sys.argv[1])
out = {}
def session():
    s = Session()
    s.upload(d["V"], d["probe"], d["prop"], sigma=float(d["sigma"]), potential_pixelsize=float(d["dz"]),
             scan_x=d["sx"], scan_y=d["sy"], measured=d["meas"], step_size=tuple(d["step"]), slice_binning=int(d["b"]))
    return s
with session() as s:
    out.update(zip(("rvol", "probe", "sx", "sy", "err"), s.run(1)))
with session() as s:
    f = s.step02(1, float(d["sx"][1]), float(d["sy"][1]))
    g = s.step03()
    out.update(waves=f["waves"], resi=f["resi"], grad=g["grad"])
np.savez(sys.argv[2], **out)
"""


@pytest.fixture(scope="module")
def deny(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("deny") / "deny_malloc.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "deny_malloc.c"), "-ldl"], check=True)
    return so


@pytest.mark.parametrize("n", [24, 32, 64, 160])
def test_pass_without_scratch_equals_pass_with_it(gpu_available, tmp_path, deny, n):
    nz, b = 5, 2
    c = small_case(n=n, nz=nz, npos=3, b=b, seed=n, defocus=20.0, jitter=4.0, strength=STRENGTH)
    np.savez(tmp_path / "in.npz", step=reasonable_steps(c), **c)
    # partial sums: doubles per warp of the field, two per position and one more
    # (the slabs are as large as another buffer of the steps)
    warps = n * {24: 8, 32: 8, 64: 8, 160: 16}[n] // 32
    sizes = f"{8 * warps * (2 * 3 + 1)},{8 * warps * 3},"
    outs = []
    for env in (dict(os.environ), dict(os.environ, LD_PRELOAD=deny, MSET_DENY_BYTES=sizes)):
        path = str(tmp_path / f"out{len(outs)}.npz")
        subprocess.run([sys.executable, "-c", SCRIPT, str(tmp_path / "in.npz"), path], check=True, env=env,
                       cwd=os.path.dirname(HERE), timeout=300)
        outs.append(dict(np.load(path)))
    a, o = outs
    for k, base in (("rvol", c["V"]), ("probe", c["probe"])):
        assert rel_l2(o[k] - base, a[k] - base) < 1e-5, k
    d = np.r_[a["sx"] - c["sx"], a["sy"] - c["sy"]]
    assert rel_l2(np.r_[o["sx"] - c["sx"], o["sy"] - c["sy"]], d) < coord_tol(n, np.r_[c["sx"], c["sy"]], d)
    assert abs(o["err"] - a["err"]) <= 1e-5 * a["err"]
    for k in ("waves", "resi", "grad"):
        assert rel_l2(o[k], a[k]) < 1e-5, k
