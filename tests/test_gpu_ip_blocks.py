"""The block kernels of incoherence processing at the edges of their 128 x 128 blocks: small and mixed transform sizes, ragged
last blocks, both layouts, and results written over their input."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(16, 16), (16, 144), (48, 80), (32, 2064), (128, 128), (112, 128), (256, 64), (144, 1040), (1040, 272), (384, 4096)]


def _reference(q, w, sv, su, cb_rms):
    """The recipe in fp64 on the CPU."""
    z = w.double() * sv.double()[:, None] * su.double()[None, :]
    out_s = z.square().mean(dim=1).sqrt().clamp_min(1e-8)
    out_s /= out_s.mean()
    z = q.block_hadamard(z / out_s[:, None], 0, 128)
    in_s = z.square().mean(dim=0).sqrt().clamp_min(1e-8)
    in_s /= in_s.mean()
    z = q.block_hadamard(z / in_s[None, :], 1, 128)
    scale = z.square().mean().sqrt() / cb_rms
    return z / scale, out_s, in_s, scale


def _rel(a, b):
    return float((a.double().cpu() - b).norm() / b.norm())


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("offset", [0, 1])
def test_forward_and_restore_match_fp64(n, k, offset):
    from trellis_b200 import _lib, qtip as q
    lib, stream, cb_rms = _lib.lib(), torch.cuda.current_stream().cuda_stream, 0.93
    g = torch.Generator().manual_seed(n * 10007 + k)
    w = torch.randn(n, k, generator=g) * torch.rand(n, 1, generator=g).add(0.1) * torch.rand(1, k, generator=g).add(0.1)
    sv, su = (torch.randint(0, 2, (d,), generator=g).float() * 2 - 1 for d in (n, k))
    z_ref, out_ref, in_ref, scale_ref = _reference(q, w, sv, su, cb_rms)
    # w may start anywhere on a 4-byte boundary, and so may the restored matrix
    store = torch.empty(n * k + offset, device="cuda")
    wd = store[offset:].view(n, k).copy_(w)
    sv, su = sv.cuda(), su.cuda()
    out_s, in_s, scale = torch.empty(n, device="cuda"), torch.empty(k, device="cuda"), torch.empty(1, device="cuda")
    ws = torch.empty(int(lib.tcq_ip_workspace_bytes(n, k)), dtype=torch.uint8, device="cuda")

    def forward(dst, tiled):
        assert lib.tcq_ip_forward(wd.data_ptr(), n, k, sv.data_ptr(), su.data_ptr(), cb_rms, tiled, dst.data_ptr(), out_s.data_ptr(),
                                  in_s.data_ptr(), scale.data_ptr(), ws.data_ptr(), ws.numel(), stream) == 0

    def restore(src, tiled, dst):
        assert lib.tcq_ip_restore(src.data_ptr(), tiled, n, k, sv.data_ptr(), su.data_ptr(), out_s.data_ptr(), in_s.data_ptr(),
                                  scale.data_ptr(), dst.data_ptr(), ws.data_ptr(), ws.numel(), stream) == 0

    rows, tiles = torch.empty(n, k, device="cuda"), torch.empty(n * k // 256, 256, device="cuda")
    forward(rows, 0)
    forward(tiles, 1)
    # fourteen butterflies and eight factors, each rounded once: 22 * 2^-24 of the norm at most
    bound = 22 * 2.0 ** -24
    assert _rel(rows, z_ref) < bound and _rel(out_s, out_ref) < bound and _rel(in_s, in_ref) < bound
    assert abs(float(scale) / float(scale_ref) - 1) < bound
    assert torch.equal(q.from_tiles(tiles, n, k), rows)
    for src, tiled in ((rows, 0), (tiles, 1)):
        back = torch.empty(n * k + offset, device="cuda")[offset:].view(n, k)
        restore(src, tiled, back)
        assert _rel(back, w.double()) < 2 * bound
        over = src.clone()                                      # results over their input
        restore(over, tiled, over)
        assert torch.equal(over.reshape(n, k), back)
    if offset == 0:
        for dst, tiled in ((rows, 0), (tiles, 1)):
            wd.copy_(w)
            forward(wd, tiled)
            assert torch.equal(wd.reshape(-1), dst.reshape(-1))
