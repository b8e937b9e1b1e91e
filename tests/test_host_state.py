"""Host code of the library that no device can be made to reach: on a CUDA
runtime of host memory (hostcuda.py)."""
import pytest

from mset_b200 import MSET_E_CUDA, MSET_E_NOMEM, MSET_E_STATE
from tests import hostcuda


def test_a_wait_that_gave_up_in_a_forward_step_is_that_call_s_error():
    r = hostcuda.run("""
s = sequential(64)
word = (C.c_uint * 1).from_address(F.fake_alloc(0))  # the session's fault word, its first allocation
word[0] = 1                                          # as the forward's kernel would leave it
report(forward=outcome(s.step02, 0, 32.0, 32.0), adjoint=outcome(s.step03), word=word[0],
       again=outcome(s.step02, 0, 32.0, 32.0), then=outcome(s.step03))
""")
    assert r["forward"][0] == MSET_E_CUDA
    assert r["adjoint"][0] == MSET_E_STATE  # no forward to go back from
    assert r["word"] == 0 and r["again"] == 0 and r["then"] == 0


def test_the_error_of_a_wait_names_what_may_have_been_waited_for():
    r = hostcuda.run("""
s = sequential(64)
(C.c_uint * 1).from_address(F.fake_alloc(0))[0] = 1
report(run=outcome(s.run, 1))
""")
    assert r["run"][0] == MSET_E_CUDA
    assert "bulk copy" in r["run"][1] and "cluster" in r["run"][1]


# (n3, n2, n1), FISTA, kernel of an iteration, launches of it in 5 iterations: few
# slices per CTA and a column per thread run in one cluster launch, more on the
# marching kernel, rows of other lengths in the cluster up to 16 columns of
# slices per thread, else on two kernels
TV_ROUTES = [
    ((24, 24, 24), True, "k_tv_cluster", 1), ((48, 24, 24), True, "k_tv_cluster", 1),
    ((64, 24, 24), True, "k_tv_march", 5), ((64, 24, 24), False, "k_tv_cluster", 1),
    ((96, 24, 24), True, "k_tv_march", 5), ((96, 24, 24), False, "k_tv_march", 5),
    ((64, 16, 16), True, "k_tv_cluster", 1), ((128, 16, 16), True, "k_tv_march", 5),
    ((32, 32, 32), True, "k_tv_march", 5), ((32, 32, 32), False, "k_tv_march", 5),
    ((8, 48, 48), True, "k_tv_march", 5), ((6000, 4, 4), True, "k_tv_march", 5),
    ((128, 128, 128), True, "k_tv_march", 5),
    ((30, 30, 30), True, "k_tv_cluster", 1), ((34, 34, 34), True, "k_tv_cluster", 1),
    ((200, 9, 9), True, "k_tv_cluster", 1), ((500, 6, 6), True, "k_tv_step", 5),
    ((4000, 5, 5), False, "k_tv_step", 5), ((60, 50, 50), True, "k_tv_step", 5),
]


def test_tv_runs_on_the_route_that_measured_fastest():
    r = hostcuda.run("""
got = []
with Session() as s:
    for shape, fista in %r:
        F.fake_clear_log()
        s.tv(np.zeros(shape, np.float32), 0.1, 5, fista)
        got.append(launched())
report(got=got, bad=F.fake_bad())
""" % [(shape, fista) for shape, fista, _, _ in TV_ROUTES])
    assert r["bad"] == 0
    for (shape, fista, kernel, launches), names in zip(TV_ROUTES, r["got"]):
        assert sum(kernel in x for x in names) == launches, (shape, fista, names)
        per_iteration = ("k_tv_cluster", "k_tv_march", "k_tv_step")
        assert sum(any(k in x for k in per_iteration) for x in names) == launches, (shape, fista, names)


def test_rotations_of_a_group_never_shear_along_the_contiguous_axis():
    """a rotation about a volume axis leaves one axis unsheared, x among the
    rows or the work volume's own fastest one: whatever else is in its group, its
    shears run along strided axes (planes that hold the contiguous one)"""
    r = hostcuda.run("""
class Job(C.Structure):  # ShearJob of csrc/mset_rotate.cu
    _fields_ = [("S", C.c_void_p), ("cx", C.c_double), ("cy", C.c_double), ("sx", C.c_int), ("sy", C.c_int),
                ("sc", C.c_int), ("real", C.c_int)]
n, turns = 24, [(0, 1), (1, 0), (2, 1), (0, 2), (1, 2)]  # (angle that is not zero, its sign or size)
b = batched(32, [1] * 6, nz=n)
ang = np.zeros((6, 3), np.float32)
for j, axis in enumerate((0, 1, 2, 1, 0, 2)):
    ang[j, axis] = 10.0  # one sub-rotation
b.iteration_setup(n, ang, positivity=False)
F.fake_watch(b"k_shear", 16 * C.sizeof(Job))
F.fake_clear_log()
b.iterate(1, use_graph=False)
strides = []
for i in range(F.fake_launches()):
    if b"k_shear" in F.fake_name(i):
        jobs = (Job * 16).from_address(F.fake_arg(i))
        strides.append([j.sc for j in jobs[:F.fake_blocks(i) // n]])
b.close()
report(strides=strides, bad=F.fake_bad())
""")
    assert r["bad"] == 0
    jobs = [s for launch in r["strides"] for s in launch]
    assert len(jobs) == 2 * 6 * 3  # there and back, six tilts, three shears that move anything
    assert 1 not in jobs


def test_sequential_pass_without_memory_for_its_slabs_runs_on_one_cta():
    r = hostcuda.run("""
got = {}
for n in (24, 32, 48, 64, 96, 128, 160, 256):
    s = sequential(n)
    F.fake_clear_log()
    F.fake_deny(n * n * 4 * 8)  # the slabs, [ns = 4][n][n] complex64
    got[n] = [outcome(s.run, 1), outcome(s.step02, 0, n / 2.0, n / 2.0)]
    F.fake_deny(8 * 3 * n * (8 if n in (24, 32, 64) else 16) // 32)  # one position's partial sums
    got[n] += [outcome(s.step03), launched()]
    F.fake_deny(0)
    s.close()
report(got=got)
""")
    for n, (run, forward, adjoint, names) in r["got"].items():
        assert (run, forward, adjoint) == (0, 0, 0), n
        assert sum("k_positions" in x for x in names) == 3 and not any("k_sequential" in x for x in names), n


def test_a_device_without_clusters_of_16_is_no_error():
    """the query for them fails there: the smaller cluster, or one CTA, runs
    and the query's error is not taken for a later launch's"""
    r = hostcuda.run("""
F.fake_clusters(-1)
s = sequential(96)
got = [s.sequential_split(), outcome(s.run, 1), outcome(s.tv, np.zeros((16, 16, 16), np.float32), 0.1, 2, True),
       outcome(s.tv, np.zeros((48, 48, 48), np.float32), 0.1, 2, True)]
report(got=got, names=launched())
""")
    assert r["got"] == [1, 0, 0, 0]
    assert any("k_tv_cluster" in x for x in r["names"]) and not any("k_sequential" in x for x in r["names"])


# an iterating session of side `edge`, and other calls on it in between
ITERATING = """
def iterating(edge, window, tilts=3):
    b = batched(window, [1] * tilts, nz=edge)
    b.iteration_setup(edge, 10.0 * np.arange(3 * tilts, dtype=np.float32).reshape(tilts, 3) + 7, positivity=False,
                      tv_lambda=0.1, tv_iter=2, tv_fista=True)
    return b

def tv(b, *shape):
    b._lib.mset_tv(b._h, flat(*shape).ctypes.data_as(C.POINTER(C.c_float)), shape[2], shape[1], shape[0], 0.1, 2, 1, None)

def rotate(b, n):
    f = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))
    v, e = flat(n, n, n), np.eye(3, dtype=np.float32)
    return b._lib.mset_rotate_volume(b._h, f(v), f(v), n, f(e[0].copy()), f(e[1].copy()), f(e[2].copy()), 0.0, 20.0, 0.0, 0)

class Job(C.Structure):  # ShearJob of csrc/mset_rotate.cu
    _fields_ = [("S", C.c_void_p), ("cx", C.c_double), ("cy", C.c_double), ("sx", C.c_int), ("sy", C.c_int),
                ("sc", C.c_int), ("real", C.c_int)]

def stale(n):
    "shears of side n that were handed a work volume outside live memory"
    live = [(F.fake_alloc(i), F.fake_alloc_bytes(i)) for i in range(F.fake_allocs())]
    bad = 0
    for i in range(F.fake_launches()):
        if b"k_shear" in F.fake_name(i):
            for j in (Job * 16).from_address(F.fake_arg(i))[:F.fake_blocks(i) // n]:
                bad += not any(p <= j.S and j.S + 8 * n ** 3 <= p + m for p, m in live)
    return bad

F.fake_watch(b"k_shear", 16 * C.sizeof(Job))
"""


@pytest.mark.parametrize("graph", [False, True], ids=["launches", "graph"])
@pytest.mark.parametrize("between", ["tv(b, 24, 24, 24)", "tv(b, 64, 64, 64)", "rotate(b, 24)", "rotate(b, 96)",
                                     "(tv(b, 50, 50, 60), rotate(b, 64), tv(b, 8, 8, 8))"])
def test_iterations_keep_their_buffers_whatever_runs_between(between, graph):
    r = hostcuda.run(ITERATING + f"""
b = iterating(48, 48)
b.iterate(1, use_graph={graph})
{between}
F.fake_clear_log()
before = F.fake_bad()
b.iterate(1, use_graph={graph})
report(before=before, bad=F.fake_bad(), stale=stale(48), n=F.fake_launches())
""")
    assert r == dict(before=0, bad=0, stale=0, n=r["n"]) and r["n"] > 10


def test_twiddles_of_the_iteration_s_side_are_back_after_another_rotation():
    r = hostcuda.run(ITERATING + """
b = iterating(48, 48)
b.iterate(1, use_graph=False)
tw = {n: np.exp(-2j * np.pi * np.outer(np.arange(n // 16), np.arange(16)) / n).astype(np.complex64) for n in (48,)}
def tables():
    "live allocations that start with the side's table [k2][n1]"
    want, m = tw[48].ravel(), 0
    for i in range(F.fake_allocs()):
        if F.fake_alloc_bytes(i) == want.nbytes:
            got = np.frombuffer((C.c_char * want.nbytes).from_address(F.fake_alloc(i)), np.complex64)
            m += np.allclose(got, want, atol=1e-6)
    return m
first = tables()
rotate(b, 64)
b.iterate(1, use_graph=False)
report(first=first, after=tables())
""")
    assert r["first"] > 0 and r["after"] == r["first"]


def test_a_setup_that_failed_half_way_leaves_nothing_to_iterate():
    r = hostcuda.run(ITERATING + """
b = iterating(48, 48)
F.fake_deny(8 * 48 * 24 * 24)  # the gradient sum of a smaller reconstruction, FP64
again = outcome(b.iteration_setup, (48, 24, 24), np.zeros((3, 3), np.float32))
F.fake_deny(0)
report(again=again[0], then=outcome(b.iterate, 1)[0], bad=F.fake_bad())
""")
    assert r == dict(again=MSET_E_NOMEM, then=MSET_E_STATE, bad=0)


@pytest.mark.parametrize("shape,zc", [((128, 128, 128), 5), ((96, 160, 160), 6), ((64, 256, 256), 5),
                                      ((96, 192, 192), 8), ((192, 256, 256), 15), ((1000, 8, 8), 1)])
def test_march_chunks_that_measured_fastest(shape, zc):
    r = hostcuda.run(f"""
with Session() as s:
    s.tv(np.zeros({shape}, np.float32), 0.1, 1, True)
report(blocks=[F.fake_blocks(i) for i in range(F.fake_launches()) if b"k_tv_march" in F.fake_name(i)])
""")
    n3, n2, n1 = shape
    rows = min(128 // (n1 // 4), n2)  # of a CTA
    assert r["blocks"] == [-(-n2 // rows) * -(-n3 // zc)]


def test_single_slice_sequential_pass_asks_for_one_slab():
    r = hostcuda.run("""
s = sequential(64)
F.fake_deny(64 * 64 * 4 * 8)  # [nz = 4][n][n] complex64
F.fake_clear_log()
report(run=outcome(s.run, 2), names=launched())
""")
    assert r["run"] == 0 and any("k_sequential" in x for x in r["names"])
