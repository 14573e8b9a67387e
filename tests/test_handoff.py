"""The hand-off between the two groups of warps of a walk (tcq_handoff.cuh) run by host threads under the thread sanitizer."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def handoff(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("handoff") / "handoff")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++20", "-O2", "-g", "-fsanitize=thread", "-isystem", os.path.join(cuda, "include"), "-o", exe,
                           os.path.join(ROOT, "tests", "handoff.cpp"), "-pthread"])
    return lambda what: subprocess.run([exe, what], capture_output=True, text=True, timeout=300)


def test_what_was_written_before_the_count_is_there(handoff):
    r = handoff("order")
    assert r.returncode == 0 and "data race" not in r.stderr, r.stderr[:2000]


def test_all_threads_leave_a_wait_with_the_same_outcome(handoff):
    """The clock of one follower runs out; the other, whose clock does not, then sees the count and still has to give up with it."""
    r = handoff("limit")
    assert r.returncode == 0 and "data race" not in r.stderr, r.stdout + r.stderr[:2000]
