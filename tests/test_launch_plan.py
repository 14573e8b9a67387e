"""What the encoder launches, and for which batch: its host code on a made-up CUDA runtime (launch_plan.cu), no GPU needed."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    """plan("encode", K, n, bytes, ...) -> the lines printed."""
    exe = str(tmp_path_factory.mktemp("plan") / "launch_plan")
    subprocess.check_call([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-Xptxas", "-O0", "-cudart", "none",
                           "-o", exe,
                           *(os.path.join(ROOT, "tests", f) for f in ("launch_plan.cu", "launch_plan_runtime.cpp"))])

    def run(*args, **env):
        return subprocess.run([exe, *map(str, args)], env={**os.environ, **env}, check=True, capture_output=True, text=True).stdout.splitlines()

    return run


def test_a_failed_query_is_asked_again(plan):
    """An occupancy query that fails says nothing about the device: the next call asks again and runs on clusters."""
    for fails in (1, 2, 5):
        lines = plan("fail", fails, *("encode", 3, 64, 0) * (fails + 1))
        calls = " ".join(lines).split("status 0")
        assert len(calls) == fails + 2
        assert "cluster" in calls[fails] and "cta" not in calls[fails]
