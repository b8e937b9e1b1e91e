"""Host code of the library that no device can be made to reach: on a CUDA
runtime of host memory (hostcuda.py)."""
from mset_b200 import MSET_E_CUDA, MSET_E_STATE
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
