"""Sweeps with fused candidates (batches of 149 tiles and more at K = 3 and 4): the square and the sum are one operation there, and the walk
and a second kernel see to it that the codes are those of the rounded operations.  TCQ_FORWARD_KERNEL=cluster2 runs every
batch with the rounded operations; the two must agree bit for bit, whatever the tiles."""
import os
import subprocess

import numpy as np
import pytest
import torch

from conftest import ROOT, same_bits

NAMES = ("1mad", "3inst", "mcg")


def _tiles(n, lut, seed):
    """Tiles of every kind by turns: Gaussian at several scales, coarse grids and few levels (ties and near-ties everywhere), zero,
    constant and periodic tiles, the codebook's own values, beyond its range, below the normal range, sums that
    overflow, NaN and infinite weights."""
    g = torch.Generator().manual_seed(seed)
    w = torch.randn(n, 256, generator=g)
    i = torch.arange(n) % 24
    w *= torch.tensor([1.24] * 6 + [0.2, 0.01, 2.5, 30.0] + [1.24] * 14)[i][:, None]
    w[i == 10], w[i == 11] = (w[i == 10] * 4).round() / 4, w[i == 11].sign()
    w[i == 12], w[i == 13] = 0.0, 0.5
    w[i == 14, ::2] = 0.0
    w[i == 15] = lut[torch.randint(0, 65536, (int((i == 15).sum()), 256), generator=g)]
    w[i == 16], w[i == 17], w[i == 18] = w[i == 16] * 1e-20, 1e18, -1.9e19
    w[i == 19, 10], w[i == 20, 200], w[i == 21] = float("nan"), float("inf"), float("nan")
    w[i == 22, 64:] = 0.0
    w[i == 23] = w[i == 23][:, :8].repeat(1, 32)
    return w


def _both(q, monkeypatch, call):
    got = call()
    monkeypatch.setenv("TCQ_FORWARD_KERNEL", "cluster2")
    want = call()
    monkeypatch.delenv("TCQ_FORWARD_KERNEL")
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    return got


@pytest.mark.gpu
@pytest.mark.parametrize("K", (3, 4))
@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("n", (149, 300, 445, 900))       # one launch and two, one chunk and two; 450 tiles to sweep again in the last
def test_codes_are_those_of_the_rounded_operations(monkeypatch, K, name, n):
    from trellis_b200 import qtip as q
    w = _tiles(n, q.codebook_lut(name, "cpu"), 10 * n + K).cuda()
    _both(q, monkeypatch, lambda: q.encode(w, K, name, want_bits=True))
    rows, comp = w.reshape(n, 16, 16).permute(2, 0, 1).reshape(16, 16 * n).contiguous(), torch.randn(16, 16 * n, device="cuda") * 0.05

    def row_block():
        wq, err = torch.empty_like(rows), torch.empty_like(rows)
        packed, sse = torch.empty(n, 8 * K, dtype=torch.int32, device="cuda"), torch.empty(n, device="cuda")
        q.encode_rows(rows, comp, K, name, wq, err, packed, sse)
        return wq, err, packed, sse

    _both(q, monkeypatch, row_block)


@pytest.mark.gpu
@pytest.mark.parametrize("K", (3, 4))
def test_a_chunk_that_leaves_a_few_tiles_over(monkeypatch, K):
    """112 tiles over, in the fused shapes of one and two tiles a cluster (900 above leave 12)."""
    test_codes_are_those_of_the_rounded_operations(monkeypatch, K, "mcg", 1000)


@pytest.mark.gpu
@pytest.mark.parametrize("K", (3, 4))
def test_a_large_batch_of_ordinary_tiles(oracle, luts, monkeypatch, K):
    """20 000 Gaussian tiles (some hundred of them with another path within the limit), and a sample against the oracle."""
    from trellis_b200 import qtip as q
    w = torch.randn(20000, 256, generator=torch.Generator().manual_seed(K)) * 1.24
    got = _both(q, monkeypatch, lambda: q.encode(w.cuda(), K, "mcg", want_bits=True))
    idx = np.arange(0, 20000, 500)
    bits, dq, sse = oracle.viterbi_tb(w.numpy()[idx], K, luts["mcg"], with_sse=True)
    assert np.array_equal(got.bits.cpu().numpy()[idx], bits) and same_bits(got.dq.cpu().numpy()[idx], dq) and same_bits(got.sse.cpu().numpy()[idx], sse)


@pytest.mark.gpu
@pytest.mark.parametrize("K", (2, 3, 4))
@pytest.mark.parametrize("n", (100, 300, 1000))
def test_the_reconstruction_may_take_the_weights_place(K, n):
    """dq over w, with tiles that are swept again among the others, at full scratch and (paths walked in parts) at little."""
    from trellis_b200 import qtip as q
    w, lib = _tiles(n, q.codebook_lut("mcg", "cpu"), n + K).cuda(), q._lib.lib()
    want = q.encode(w, K, "mcg")
    for ws_bytes in (int(lib.tcq_workspace_bytes(n, K)), n // 5 * int(lib.tcq_workspace_min_bytes(K))):
        ws, x = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda"), w.clone()
        packed, sse = torch.zeros(n, 8 * K, dtype=torch.int32, device="cuda"), torch.zeros(n, device="cuda")
        assert lib.tcq_encode_tb(x.data_ptr(), n, K, 2, packed.data_ptr(), None, x.data_ptr(), sse.data_ptr(), ws.data_ptr(), ws_bytes,
                                 torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(packed, want.packed) and torch.equal(x.view(torch.int32), want.dq.view(torch.int32))
        assert torch.equal(sse.view(torch.int32), want.sse.view(torch.int32))


def _listed(ws):
    """How many tiles the walks of the two passes of a span have listed (the words that tcq_capi.cu's `counts` names)."""
    return ws[16:24].view(torch.int32).tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("K", (3, 4))
@pytest.mark.parametrize("n,size_for", ((700, 350), (1000, 888), (2700, 888)))         # two spans, two with a short one, four
def test_batches_of_several_spans(monkeypatch, K, n, size_for):
    """Scratch sized for fewer tiles: the lists, the overlaps and the counts of a span are those of the span before, used again."""
    from trellis_b200 import qtip as q
    lib = q._lib.lib()
    w = _tiles(n, q.codebook_lut("1mad", "cpu"), n + K).cuda()
    ws = torch.full((int(lib.tcq_workspace_bytes(size_for, K)),), 0x5A, dtype=torch.uint8, device="cuda")

    def encode():
        packed, dq, sse = torch.zeros(n, 8 * K, dtype=torch.int32, device="cuda"), torch.zeros(n, 256, device="cuda"), torch.zeros(n, device="cuda")
        assert lib.tcq_encode_tb(w.data_ptr(), n, K, 0, packed.data_ptr(), None, dq.data_ptr(), sse.data_ptr(), ws.data_ptr(), ws.numel(),
                                 torch.cuda.current_stream().cuda_stream) == 0
        return packed, dq, sse

    _both(q, monkeypatch, encode)


@pytest.mark.gpu
@pytest.mark.parametrize("K", (3, 4))
def test_what_the_walk_settles_and_what_it_lists(K):
    """Of 20 000 Gaussian tiles 400 have a second edge at the end of pass 1, a hundred or two a marked node in a pass and some twenty are walked back to the beginning:
    no more than a few are listed, so each of these is settled and not left to the second sweep.  Tiles whose costs are above 1e37 are all listed
    (of ties alone that does not hold in both passes: over zeros the free pass has one best path)."""
    from trellis_b200 import qtip as q
    lib, stream = q._lib.lib(), torch.cuda.current_stream().cuda_stream
    for w, least, most in ((torch.randn(20000, 256, generator=torch.Generator().manual_seed(K)) * 1.24, 0, 20), (torch.full((300, 256), 1e18), 300, 300)):
        n, w = w.shape[0], w.cuda()
        ws, packed = torch.zeros(int(lib.tcq_workspace_bytes(n, K)), dtype=torch.uint8, device="cuda"), torch.zeros(n, 8 * K, dtype=torch.int32, device="cuda")
        assert lib.tcq_encode_tb(w.data_ptr(), n, K, 2, packed.data_ptr(), None, None, None, ws.data_ptr(), ws.numel(), stream) == 0
        assert all(least <= x <= most for x in _listed(ws)), _listed(ws)


@pytest.mark.gpu
@pytest.mark.parametrize("K", (3, 4))
@pytest.mark.parametrize("n", (200, 296, 370, 444))       # three to six tiles a cluster
def test_single_passes_keep_the_rounded_shapes(K, n):
    """tcq_viterbi_pass sweeps every batch with rounded operations; its two passes give the codes of an encode."""
    from trellis_b200 import qtip as q
    w = (torch.randn(n, 256, generator=torch.Generator().manual_seed(n + K)) * 1.24).cuda()
    overlap = (q.viterbi_pass_b200(w, K, None, "mcg", roll=128)[:, 128] >> K).int()
    states = q.viterbi_pass_b200(w, K, overlap, "mcg")
    assert torch.equal(states & (2 ** K - 1), q.encode(w, K, "mcg", want_bits=True).bits)


@pytest.mark.gpu
@pytest.mark.parametrize("K", (3, 4))
def test_a_walk_that_does_not_wait_lists_its_tile(K):
    """The second group of warps gives up at once where the first has not come far enough, now one warp of it first and now the other: the
    tiles are swept again, nothing hangs, and the codes are the same."""
    from trellis_b200 import qtip as q
    n, lib = 600, q._lib.lib()
    w = (torch.randn(n, 256, generator=torch.Generator().manual_seed(K)) * 1.24).cuda()
    ws = torch.zeros(int(lib.tcq_workspace_bytes(n, K)), dtype=torch.uint8, device="cuda")
    stream, want, got = torch.cuda.current_stream().cuda_stream, *torch.zeros(2, n, 8 * K, dtype=torch.int32, device="cuda")
    assert lib.tcq_encode_tb(w.data_ptr(), n, K, 2, want.data_ptr(), None, None, None, ws.data_ptr(), ws.numel(), stream) == 0
    assert max(_listed(ws)) <= n // 100
    for _ in range(5):
        got.zero_()
        assert lib.tcq_selftest_walk_waits(w.data_ptr(), n, K, got.data_ptr(), ws.data_ptr(), ws.numel(), stream) == 0
        assert torch.equal(got, want) and min(_listed(ws)) > n // 2
    assert lib.tcq_workspace_status(ws.data_ptr(), ws.numel(), n, K, stream) == 0


def test_the_bound_between_fused_and_rounded_sums():
    """|A - F| <= (2 t + 2) u H of the limit (fused_limit), over random, repeated and graded terms; A as the fused operation gives it (the
    square is exact in 64 bits, the sum there rounds 2^29 times finer)."""
    rng = np.random.default_rng(1)
    for d in (rng.normal(size=(256, 2000)), np.repeat(rng.normal(size=(1, 2000)), 256, 0), rng.normal(size=(256, 2000)) * np.logspace(-4, 2, 256)[:, None],
              np.tile(rng.normal(size=(8, 2000)), (32, 1)) * 0.17, rng.normal(size=(256, 2000)) ** 9):
        d = d.astype(np.float32)
        A, F = np.zeros(2000, np.float32), np.zeros(2000, np.float32)
        for t in range(256):
            A = (d[t].astype(np.float64) ** 2 + A).astype(np.float32)
            F = d[t] * d[t] + F
            H = 2.0 ** np.floor(np.log2(np.maximum((A * np.float32(1.0005)).astype(np.float64), 1e-30)))
            assert (np.abs(A.astype(np.float64) - F) <= (2 * (t + 1) + 2) * 2.0 ** -24 * H).all()


@pytest.fixture(scope="module")
def fused_limit(tmp_path_factory):
    """fused_limit of tcq_walk.cuh: (smallest candidates, steps) -> limits."""
    exe = str(tmp_path_factory.mktemp("limit") / "fused_limit")
    subprocess.check_call([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-fmad=false",
                           "-o", exe, os.path.join(ROOT, "tests", "fused_limit.cu")])

    def run(best, t):
        pairs = np.empty(best.size, [("best", np.float32), ("t", np.int32)])
        pairs["best"], pairs["t"] = best.ravel(), t.ravel()
        return np.frombuffer(subprocess.run([exe], input=pairs.tobytes(), check=True, capture_output=True).stdout, np.float32).reshape(best.shape)

    return run


def test_the_limit_holds_the_bound_between_fused_and_rounded_sums(fused_limit):
    """|A - F| <= (2 t + 2) u H, and no more than half of what fused_limit adds, so that of two candidates one of which is beyond the other's limit
    that one is the larger by the rounded sums too; over random, repeated and graded terms.  A as the fused operation gives it (the
    square is exact in 64 bits, the sum there rounds 2^29 times finer).  The limit adds no more than it says."""
    rng = np.random.default_rng(1)
    for d in (rng.normal(size=(256, 2000)), np.repeat(rng.normal(size=(1, 2000)), 256, 0), rng.normal(size=(256, 2000)) * np.logspace(-4, 2, 256)[:, None],
              np.tile(rng.normal(size=(8, 2000)), (32, 1)) * 0.17, rng.normal(size=(256, 2000)) ** 9):
        d = d.astype(np.float32)
        A, F = np.zeros((256, 2000), np.float32), np.zeros((256, 2000), np.float32)
        a = f = np.zeros(2000, np.float32)
        for t in range(256):
            A[t] = a = (d[t].astype(np.float64) ** 2 + a).astype(np.float32)
            F[t] = f = d[t] * d[t] + f
        steps = np.broadcast_to(np.arange(1, 257, dtype=np.int32)[:, None], A.shape)
        H = 2.0 ** np.floor(np.log2(np.maximum((A * np.float32(1.0005)).astype(np.float64), 1e-30)))
        off = np.abs(A.astype(np.float64) - F)
        assert (off <= (2 * steps + 2) * 2.0 ** -24 * H).all()
        added = fused_limit(A, steps).astype(np.float64) - A
        assert (2 * off <= added).all()
        assert (added >= (4 * steps + 4) * 2.0 ** -24 * H).all() and (added <= (4 * steps + 18) * 2.0 ** -24 * H + 2e-30).all()
