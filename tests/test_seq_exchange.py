"""The rules of a cluster pass whose bounded wait gave up (csrc/seq_exchange.h)
on modelled mbarriers: every thread gives up in turn, and no barrier's
transaction count leaves the range it can hold."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.access("/usr/bin/g++", os.X_OK) else shutil.which("g++")
    exe = str(tmp_path_factory.mktemp("model") / "seq_exchange_model")
    subprocess.run([cxx, "-O1", "-std=c++17", "-o", exe, os.path.join(HERE, "seq_exchange_model.cpp")], check=True)
    return exe


@pytest.mark.parametrize("cta,thread,at", [(0, 0, 5), (3, 7, 5), (3, 0, 6), (15, 31, 6), (1, 16, 399)])
def test_a_thread_that_gives_up_ends_the_exchanges(model, cta, thread, at):
    total = 400
    out = subprocess.run([model, str(cta), str(thread), str(at), str(total)], check=True, capture_output=True, text=True)
    worst, dead = map(int, out.stdout.split())
    assert worst < 2 ** 20
    assert dead == (16 * 32 if at + 3 < total else 1)


def test_without_a_failure_nobody_gives_up(model):
    out = subprocess.run([model, "0", "0", "400", "400"], check=True, capture_output=True, text=True)
    worst, dead = map(int, out.stdout.split())
    assert worst <= 32768 and dead == 0
