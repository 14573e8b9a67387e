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
    return lambda: subprocess.run([exe], capture_output=True, text=True, timeout=300)


def test_what_was_written_before_the_count_is_there(handoff):
    r = handoff()
    assert r.returncode == 0 and "data race" not in r.stderr, r.stderr[:2000]
