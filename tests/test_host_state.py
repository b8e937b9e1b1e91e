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
