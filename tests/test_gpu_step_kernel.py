"""The cluster step kernel and the walk over its metric rows: every launch shape, every way a workspace can be cut, and
inputs on which candidates tie or are not numbers.  The codec's results are exact, so all comparisons are bit for bit."""
import numpy as np
import pytest
import torch

from conftest import KS, same_bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def q():
    from trellis_b200 import qtip
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    qtip._lib.lib()
    return qtip


def _np(t):
    return t.detach().cpu().numpy()


# one tile, and both sides of every batch size up to two rounds of the largest shape at which another shape (SMs per cluster x tiles
# per cluster) takes over (test_launch_plan.py holds them against the plan); some go as two launches, whole rounds of one shape and the
# rest in another
_ROUNDS = tuple(m for k in range(1, 12) for m in (74 * k, 74 * k + 1))
SIZES = {2: (1, 7, 8, 9, 15, 16, 17, 30, 31, 33, 34, 67, 299, 671, 888) + _ROUNDS, 3: (1, 15, 16, 17, 30, 31, 32, 33, 34, 66, 67, 443, 768, 888) + _ROUNDS,
         4: (1, 15, 16, 17, 33, 34, 67, 521, 888) + _ROUNDS}


@pytest.mark.parametrize("K,n", [(K, n) for K in KS for n in SIZES[K]])
def test_every_launch_shape_matches_the_oracle(q, oracle, luts, K, n):
    name = ("1mad", "3inst", "mcg")[n % 3]
    w = torch.randn(n, 256, generator=torch.Generator().manual_seed(1000 * K + n)) * 1.1
    r = q.encode(w.cuda(), K, name, want_bits=True)
    idx = np.unique(np.concatenate((np.arange(min(n, 8)), np.arange(max(n - 8, 0), n), np.arange(0, n, 29))))
    bits, dq, sse = oracle.viterbi_tb(w.numpy()[idx], K, luts[name], with_sse=True)
    assert np.array_equal(_np(r.bits)[idx], bits)
    assert same_bits(_np(r.dq)[idx], dq) and same_bits(_np(r.sse)[idx], sse)
    assert np.array_equal(_np(r.packed)[idx].view(np.uint32), oracle.pack_bits(bits, K))
    q.workspace_status(n, K)


@pytest.mark.parametrize("K", KS)
def test_workspaces_of_every_size_give_the_same_codes(q, K):
    """From the smallest accepted scratch (rows of a quarter of the path of one tile) over halves to whole paths; tiles,
    row blocks and single passes."""
    lib = q._lib.lib()
    n, nw = 21, 8 * K
    w = torch.randn(n, 256, device="cuda")
    rows = torch.randn(16, 16 * n, device="cuda")
    comp = torch.randn(16, 16 * n, device="cuda") * 0.1
    stream = torch.cuda.current_stream().cuda_stream
    per_tile = int(lib.tcq_workspace_min_bytes(K))
    ref = None
    for ws_bytes in (per_tile, 2 * per_tile - 4096, 5 * per_tile + 12345, 12 * per_tile, n * per_tile, int(lib.tcq_workspace_bytes(n, K))):
        ws = torch.full((ws_bytes,), 0xA5, dtype=torch.uint8, device="cuda")
        packed, bits = torch.zeros(n, nw, dtype=torch.int32, device="cuda"), torch.zeros(n, 256, dtype=torch.int64, device="cuda")
        dq, sse = torch.zeros(n, 256, device="cuda"), torch.zeros(n, device="cuda")
        args = (ws.data_ptr(), ws_bytes, stream)
        assert lib.tcq_encode_tb(w.data_ptr(), n, K, 1, packed.data_ptr(), bits.data_ptr(), dq.data_ptr(), sse.data_ptr(), *args) == 0
        assert lib.tcq_workspace_status(ws.data_ptr(), ws_bytes, n, K, stream) == 0
        wq, err, rpacked, rsse = torch.zeros_like(rows), torch.zeros_like(rows), torch.zeros_like(packed), torch.zeros_like(sse)
        assert lib.tcq_encode_tb_rows(rows.data_ptr(), comp.data_ptr(), 16 * n, 16 * n, K, 2, rpacked.data_ptr(), nw, wq.data_ptr(),
                                      err.data_ptr(), rsse.data_ptr(), *args) == 0
        states = torch.zeros(n, 256, dtype=torch.int64, device="cuda")
        assert lib.tcq_viterbi_pass(w.data_ptr(), n, K, 0, None, 128, states.data_ptr(), *args) == 0
        out = (packed, bits, dq, sse, wq, err, rpacked, rsse, states)
        torch.cuda.synchronize()
        if ref is None:
            ref = out
            assert int(lib.tcq_encode_launches(n, K, ws_bytes)) > 4 * n          # parts: more than one sweep per pass
        for a, b in zip(ref, out):
            assert torch.equal(a, b)
    assert int(lib.tcq_encode_launches(n, K, ws_bytes)) == 4
    assert int(lib.tcq_encode_launches(223, K, int(lib.tcq_workspace_bytes(223, K)))) in (4, 6)      # a sweep may be two launches
    small = torch.empty(per_tile, dtype=torch.uint8, device="cuda")
    assert lib.tcq_encode_tb(w.data_ptr(), n, K, 1, packed.data_ptr(), None, None, None, small.data_ptr(), per_tile - 1, stream) == -6


def test_a_nearly_full_device_encodes_with_less_scratch(q):
    """768 tiles at K = 3 ask for 2.1 GB of scratch; where 1.2 GB are left the call runs on less, with the same results and status."""
    n, K = 768, 3
    w = torch.randn(n, 256, generator=torch.Generator().manual_seed(3)).cuda()
    want = q.encode(w, K, "mcg")
    q.release_workspaces()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 1.2e9) / total)
    try:
        got = q.encode(w, K, "mcg")
        q.workspace_status(n, K)
        w[5, 5] = float("nan")
        q.encode(w, K, "mcg")
        with pytest.raises(q._lib.TcqError, match="NaN"):
            q.workspace_status(n, K)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        q.release_workspaces()
    assert all(torch.equal(a, b) for a, b in zip(got[:3], want[:3]))


@pytest.mark.parametrize("K", KS)
@pytest.mark.parametrize("name", ("1mad", "3inst", "mcg"))
def test_ties_and_numbers_that_are_none(q, K, name, monkeypatch):
    """The walk re-derives the argmins that the single-CTA kernel records as it goes: the two must choose alike where
    candidates tie (constant and zero tiles, subnormal distances, codebook values hit exactly, metrics that have absorbed every
    distance) and where none compares (NaN and infinite weights)."""
    w = torch.randn(24, 256, generator=torch.Generator().manual_seed(5))
    w[0], w[1], w[2], w[3] = 0.0, 0.5, 1e-20, -1e-38
    w[4] = q.codebook_lut(name, "cpu")[torch.arange(256) * 251]
    w[5], w[6], w[7], w[8] = 3e7, 1e18, -1.9e19, 1e30
    w[9, 10], w[10, 0], w[11, 255], w[12, 128] = float("nan"), float("inf"), float("-inf"), float("nan")
    w[13] = float("nan")
    w[14] = float("inf")
    w[15, ::2] = 0.0
    w[16] = w[16].round()
    w = w.cuda()
    r = q.encode(w, K, name, want_bits=True)
    p1 = q.viterbi_pass_b200(w, K, None, name)
    monkeypatch.setenv("TCQ_FORWARD_KERNEL", "cta")
    o = q.encode(w, K, name, want_bits=True)
    assert torch.equal(r.bits, o.bits) and torch.equal(r.packed, o.packed) and torch.equal(r.dq, o.dq)
    assert torch.equal(r.sse.view(torch.int32), o.sse.view(torch.int32))
    assert torch.equal(p1, q.viterbi_pass_b200(w, K, None, name))
