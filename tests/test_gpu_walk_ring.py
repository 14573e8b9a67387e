"""The walk with rows fetched ahead into shared memory: both sides of the batch sizes that take it, walks of whole paths and of parts
of them (rows that wrap around the ring, rows that do not fill it), against the oracle bit for bit."""
import numpy as np
import pytest
import torch

from conftest import KS, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", KS)
@pytest.mark.parametrize("n", (2, 3, 74, 75, 96, 97, 148))
def test_rows_in_the_ring(oracle, luts, K, n):
    from trellis_b200 import qtip as q
    w = torch.randn(n, 256, generator=torch.Generator().manual_seed(100 * K + n)) * 1.2
    idx = np.unique(np.concatenate((np.arange(min(n, 4)), np.arange(0, n, 37), [n - 1])))
    bits, dq, sse = oracle.viterbi_tb(w.numpy()[idx], K, luts["3inst"], with_sse=True)
    lib, stream = q._lib.lib(), torch.cuda.current_stream().cuda_stream
    wd = w.cuda()
    for ws_bytes in (int(lib.tcq_workspace_bytes(n, K)), n * int(lib.tcq_workspace_min_bytes(K))):      # whole paths, halves or quarters
        ws = torch.full((ws_bytes,), 0x5A, dtype=torch.uint8, device="cuda")
        packed, b = torch.zeros(n, 8 * K, dtype=torch.int32, device="cuda"), torch.zeros(n, 256, dtype=torch.int64, device="cuda")
        d, s = torch.zeros(n, 256, device="cuda"), torch.zeros(n, device="cuda")
        assert lib.tcq_encode_tb(wd.data_ptr(), n, K, 1, packed.data_ptr(), b.data_ptr(), d.data_ptr(), s.data_ptr(), ws.data_ptr(), ws_bytes, stream) == 0
        assert np.array_equal(b.cpu().numpy()[idx], bits)
        assert same_bits(d.cpu().numpy()[idx], dq) and same_bits(s.cpu().numpy()[idx], sse)


@pytest.mark.parametrize("K", KS)
@pytest.mark.parametrize("n", (3, 8, 74))
def test_rows_that_do_not_come_in_time(K, n):
    """The walk waits for no row: it reads them from global memory, the status word says so, and the CTA ends after its copies.
    The calls that follow on the same SMs are sound."""
    from trellis_b200 import qtip as q
    lib, stream = q._lib.lib(), torch.cuda.current_stream().cuda_stream
    w = (torch.randn(n, 256, generator=torch.Generator().manual_seed(n + K)) * 1.2).cuda()
    want = q.encode(w, K, "mcg").packed
    for ws_bytes in (int(lib.tcq_workspace_bytes(n, K)), n * int(lib.tcq_workspace_min_bytes(K))):
        ws, packed = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda"), torch.zeros(n, 8 * K, dtype=torch.int32, device="cuda")
        assert lib.tcq_selftest_walk_waits(w.data_ptr(), n, K, packed.data_ptr(), ws.data_ptr(), ws_bytes, stream) == 0
        assert lib.tcq_workspace_status(ws.data_ptr(), ws_bytes, n, K, stream) == -10          # TCQ_E_DEVICE_TIMEOUT
        assert torch.equal(packed, want)
        packed.zero_()
        assert lib.tcq_encode_tb(w.data_ptr(), n, K, 2, packed.data_ptr(), None, None, None, ws.data_ptr(), ws_bytes, stream) == 0
        assert lib.tcq_workspace_status(ws.data_ptr(), ws_bytes, n, K, stream) == 0 and torch.equal(packed, want)
