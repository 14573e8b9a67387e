"""What the encoder launches, and for which batch: its host code on a made-up CUDA runtime (launch_plan.cu), no GPU needed."""
import os
import re
import subprocess

import pytest

from conftest import KS, ROOT
from test_gpu_step_kernel import SIZES


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


def test_a_cluster_size_that_a_rate_has_not_is_refused(plan):
    """TCQ_FORWARD_KERNEL fixes the cluster size for comparison runs: what it names runs or the call is refused, and text that
    names nothing is no request."""
    for K, C in ((2, 2), (2, 8), (2, 16), (3, 2), (3, 4), (3, 8), (4, 2), (4, 4), (4, 8)):
        lines = plan("encode", K, 5, 0, TCQ_FORWARD_KERNEL=f"cluster{C}")
        assert lines[-1] == "status 0" and all(f" C={C} " in x for x in lines if x.startswith("c"))
    for K in (3, 4):
        assert plan("encode", K, 5, 0, TCQ_FORWARD_KERNEL="cluster16") == ["status -8"]
    for text in ("cluster3", "cluster", "warp"):
        assert plan("encode", 3, 5, 0, TCQ_FORWARD_KERNEL=text) == plan("encode", 3, 5, 0)
    assert any(x.startswith("cta") for x in plan("encode", 3, 5, 0, TCQ_FORWARD_KERNEL="cta"))


@pytest.mark.parametrize("K", KS)
def test_every_shape_is_some_batch_s_and_every_switch_is_tested(plan, K):
    """No shape is compiled that no batch takes, and the sizes of the GPU test hold both sides of every size at which another
    shape, or another pair of shapes, takes over (up to two rounds of the largest, the tiles of one chunk)."""
    lines = plan(*(x for n in range(1, 889) for x in ("encode", K, n, 0)))
    calls = "\n".join(lines).split("status 0")[:-1]
    taken = [tuple(re.findall(r"C=\d+ G=\d+", c)) for c in calls]
    assert {s for t in taken for s in t} == set(plan("shapes", K))
    switches = [n for n in range(2, 889) if taken[n - 1] != taken[n - 2]]
    assert len(switches) >= 10 and {n - 1 for n in switches} | set(switches) <= set(SIZES[K])


@pytest.mark.parametrize("K", KS)
def test_every_form_is_some_batch_s_and_every_switch_is_tested(plan, K):
    """No shape is compiled that no batch takes, in either form (at K = 3 and 4 the rounded shapes of three to six tiles are those of single passes, the
    fused ones of one and two those of what a chunk leaves over), and the sizes of the GPU test hold both sides of every size at which another shape, or another pair of shapes, or the other form
    takes over (up to two rounds of the largest, the tiles of one chunk)."""
    shape = re.compile(r"(C=\d+ G=\d+) .* (rounded|fused|listed)")
    of = lambda what: [[" ".join(x) for x in shape.findall(c)] for c in "\n".join(plan(*(x for n in range(1, 1037) for x in (what, K, n, 0)))).split("status 0")[:-1]]
    encodes, passes = of("encode"), of("pass")
    assert {s for t in encodes + passes for s in t} - {"C=2 G=2 listed"} == set(plan("forms", K))
    assert not any(s.endswith("rounded") for t in encodes[148:] for s in t) if K > 2 else all(s.endswith("rounded") for t in encodes for s in t)
    assert all(s.endswith("rounded") for t in passes for s in t)
    switches = [n for n in range(2, 889) if encodes[n - 1] != encodes[n - 2]]
    assert len(switches) >= 10 and {n - 1 for n in switches} | set(switches) <= set(SIZES[K])


def _earlier_size(n, K):
    """Scratch that held the recorded argmins of n tiles: a quarter to a third of what their metric rows take."""
    up = lambda b: -(-b // 256) * 256
    return up(n * 256 * (1 << (16 - K)) * K // 8) + 2 * up(4 * n) + up(32 * n) + 256


@pytest.mark.parametrize("K", KS)
def test_every_plan_stays_inside_its_scratch(plan, K):
    full = lambda n: 0
    for size in (full, lambda n: _earlier_size(n, K), lambda n: _earlier_size(n, K) // 2 + 1024 * 1024, lambda n: _earlier_size(1, K)):
        lines = plan(*(x for n in (1, 2, 7, 8, 15, 16, 17, 31, 64, 100, 101, 443, 888, 1000) for x in ("encode", K, n, size(n))))
        assert lines.count("status 0") == 14 and not [x for x in lines if x.startswith(("outside", "shared"))]
    assert not [x for x in plan("encode", 2, 100, 0, TCQ_FORWARD_KERNEL="cluster16") if x.startswith(("outside", "shared"))]


@pytest.mark.parametrize("K", (3, 4))
def test_spans_of_fused_batches_stay_inside_their_scratch(plan, K):
    """Batches that go in several spans: scratch sized for fewer tiles than the batch has."""
    for n, m, spans in ((700, 350, 2), (1000, 888, 2), (2700, 888, 4), (5000, 888, 6)):
        lines = plan("encode", K, n, int(plan("size", K, m, 0)[0]))
        walks = [int(re.search(r" n=(\d+) ", x).group(1)) for x in lines if x.startswith("walk")]
        assert lines[-1] == "status 0" and not [x for x in lines if x.startswith(("outside", "shared"))]
        assert sum(walks) == 2 * n and sum(x.endswith("listed") for x in lines) == 2 * spans


@pytest.mark.parametrize("n,tiles", [(48, 24), (64, 32), (200, 67), (256, 128), (300, 150), (444, 222)])
def test_half_paths_fit_half_the_tiles_of_the_earlier_size(plan, n, tiles):
    """K = 4: the rows of half a path are twice the argmins of a whole one, so half the tiles fit: two chunks of three walks each, the
    fastest plan for these sizes, or three where a third fits a round of a faster shape."""
    walks = [x for x in plan("encode", 4, n, _earlier_size(n, 4)) if x.startswith("walk")]
    assert len(walks) == 3 * -(-n // tiles) and f" n={tiles} " in walks[0]
