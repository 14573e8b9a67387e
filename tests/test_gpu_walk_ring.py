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
