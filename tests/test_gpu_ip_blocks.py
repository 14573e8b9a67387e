"""The kernels of incoherence processing at the edges of their 128 x 128 blocks: small and mixed transform sizes, ragged
last blocks, both layouts, and results written over their input; against fp64, and bit for bit against the same roundings in
the same order, because the packed bytes of a matrix hang on them."""
import numpy as np
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


def _halves(x):
    while x.shape[-1] > 1:
        x = x[..., :x.shape[-1] // 2] + x[..., x.shape[-1] // 2:]
    return x[..., 0]


def _mod_sums(x, m, fused_square=False):
    """Partial sums over the indices i mod m of the last axis, in index order."""
    s = np.zeros((*x.shape[:-1], m), np.float32)
    for i in range(0, x.shape[-1], m):
        b = x[..., i:i + m]
        d = b.shape[-1]
        # a product of two fp32 numbers is exact in fp64, so that the sum is rounded as a fused multiply-add rounds it
        s[..., :d] = (b.astype(np.float64) ** 2 + s[..., :d]).astype(np.float32) if fused_square else s[..., :d] + b
    return s


def _hadamard(z, axis):
    b = 1
    while b < 128 and z.shape[axis] % (2 * b) == 0:
        b *= 2
    z = np.moveaxis(z, axis, 0)
    shape = z.shape
    h = 1
    while h < b:
        p = z.reshape(-1, 2, h, shape[1])
        z = np.stack((p[:, 0] + p[:, 1], p[:, 0] - p[:, 1]), axis=1)
        h *= 2
    return np.moveaxis(z.reshape(shape), 0, axis), np.float32(1 / np.sqrt(float(b))), b


def _in_order(w, sv, su, cb_rms):
    """The forward recipe in fp32, every rounding and every sum in the library's order: z, out_s, in_s, scale."""
    f = np.float32
    n, k = w.shape

    def scales(ms, d):
        r = np.fmax(np.sqrt(ms / f(d)), f(1e-8))
        return r / (_halves(_mod_sums(r, 1024)) / f(len(r)))

    out_s = scales(_halves(_mod_sums(w, 256, fused_square=True)), k)
    z, norm, b = _hadamard(w * (sv * (f(1) / out_s))[:, None] * su, 0)
    z = z * norm
    t = np.zeros(k, f)
    for p in _mod_sums(np.moveaxis(z.reshape(n // b, b, k), 1, 2), 1, fused_square=True)[..., 0]:
        t = t + p
    in_s = scales(t, n)
    scale = np.sqrt(_halves(_mod_sums(t / (in_s * in_s), 1024)) / (f(n) * f(k))) / f(cb_rms)
    z, norm, _ = _hadamard(z * (f(1) / in_s), 1)
    return z * norm * (f(1) / scale), out_s, in_s, scale


def _back_in_order(z, sv, su, out_s, in_s, scale):
    y, norm1, _ = _hadamard(z * scale, 1)
    y, norm0, _ = _hadamard(y * norm1 * in_s, 0)
    return y * norm0 * out_s[:, None] * sv[:, None] * su


def _same(a, b):
    return np.array_equal(a.detach().cpu().numpy(), b, equal_nan=True)


def _check_bits(w, cb_rms=0.93, seed=11):
    from trellis_b200 import qtip as q
    n, k = w.shape
    ip = q.IPContext(w.cuda(), cb_rms, seed=seed)
    sv, su = ip.sv.cpu().numpy(), ip.su.cpu().numpy()
    with np.errstate(all="ignore"):
        z, out_s, in_s, scale = _in_order(w.numpy(), sv, su, cb_rms)
        assert _same(ip.out_s, out_s) and _same(ip.in_s, in_s) and _same(ip._scale_t, scale[None])
        assert _same(ip.z, z)
        back = _back_in_order(z, sv, su, out_s, in_s, scale)
    assert _same(ip.restore_tiles(ip.tiles), back) and _same(ip.restore(ip.z), back)


@pytest.mark.parametrize("n,k", SHAPES + [(64, 12288), (1184, 48), (1200, 528), (2064, 1040)])
def test_every_rounding_in_order(n, k):
    g = torch.Generator().manual_seed(n * 31 + k)
    w = torch.randn(n, k, generator=g) * torch.rand(n, 1, generator=g).add(0.1)
    _check_bits(torch.where(torch.rand(n, k, generator=g) < 0.01, w * 20, w))


@pytest.mark.parametrize("case", ["zero", "zero rows and columns", "below the clamp", "tiny", "large", "spread", "inf", "nan"])
def test_degenerate_matrices_in_order(case):
    n, k = 272, 400
    w = torch.randn(n, k, generator=torch.Generator().manual_seed(9))
    if case == "zero":
        w.zero_()
    elif case == "zero rows and columns":
        w[[0, 17, 271]], w[:, [0, 33, 399]] = 0.0, 0.0
    elif case == "below the clamp":
        w[5], w[:, 12] = w[5] * 1e-10, w[:, 12] * 1e-11
    elif case == "tiny":
        w *= 1e-12
    elif case == "large":
        w *= 1e15
    elif case == "spread":
        w *= torch.logspace(-12, 6, n)[:, None]
    elif case == "inf":
        w[3, 7] = float("inf")
    else:
        w[130, 200] = float("nan")
    _check_bits(w)
