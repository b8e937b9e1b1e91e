"""Runs a script with the library on a CUDA runtime of host memory
(fake_cudart.c): its host code really runs, its kernels are only logged.  For
what cannot be made to happen on a device (a wait that gave up, no memory left,
a buffer freed under a captured graph)."""
import json
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
_lib = None

PRELUDE = """
import ctypes as C, json, os
import numpy as np
from mset_b200 import MsetError, Session
from mset_b200.batch import BatchSession
F = C.CDLL(os.environ["LD_PRELOAD"])
F.fake_name.restype = C.c_char_p
F.fake_alloc.restype = F.fake_arg.restype = C.c_void_p
F.fake_alloc_bytes.restype = C.c_size_t
F.fake_deny.argtypes = [C.c_size_t]
F.fake_watch.argtypes = [C.c_char_p, C.c_size_t]

def launched():
    return [F.fake_name(i).decode() for i in range(F.fake_launches())]

def outcome(f, *a, **kw):
    "0, or the status and text of the error"
    try:
        f(*a, **kw)
        return 0
    except MsetError as e:
        return [e.code, str(e)]

def flat(*shape):
    return np.ones(shape, np.float32)

def sequential(n, nz=4, npos=2):
    s = Session()
    s.upload(flat(nz, n, n), flat(n, n).astype(np.complex64), flat(n, n).astype(np.complex64), sigma=1e-3,
             potential_pixelsize=0.4, scan_x=n / 2 * flat(npos), scan_y=n / 2 * flat(npos),
             measured=flat(npos, n, n), step_size=(1e-3, 1e-3, 1e-3))
    return s

def batched(n, npos, nz=4, binning=1):
    b = BatchSession(n=n, nz=nz, npos=npos, prop=flat(n, n).astype(np.complex64), sigma=1e-3,
                     potential_pixelsize=0.4, slice_binning=binning)
    for j, p in enumerate(npos):
        b.set_tilt(j, probe=flat(n, n).astype(np.complex64), scan_x=n / 2 * flat(p), scan_y=n / 2 * flat(p),
                   measured=flat(p, n, n), volume=flat(nz, n, n))
    return b

def report(**kw):
    print("RESULT" + json.dumps(kw))
"""


def fake_runtime() -> str:
    global _lib
    if _lib is None:
        _lib = os.path.join(tempfile.mkdtemp(prefix="mset_host_"), "libfake_cudart.so")
        cc = "/usr/bin/gcc" if os.access("/usr/bin/gcc", os.X_OK) else "gcc"
        subprocess.run([cc, "-O1", "-Wall", "-shared", "-fPIC", "-o", _lib, os.path.join(HERE, "fake_cudart.c")],
                       check=True)
    return _lib


def run(script: str) -> dict:
    """what the script hands to report()"""
    env = dict(os.environ, LD_PRELOAD=fake_runtime())
    r = subprocess.run([sys.executable, "-c", PRELUDE + script], env=env, cwd=os.path.dirname(HERE),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.split("RESULT", 1)[1])
