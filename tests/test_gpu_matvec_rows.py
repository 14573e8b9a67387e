"""Decode-matvec: an odd number of tile rows where a CTA has two, right-hand sides that do not fill the four, and both sides of every
number of tile rows at which another form of the kernel takes over."""
import pytest
import torch

from conftest import KS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", KS)
@pytest.mark.parametrize("m", [3, 4, 6])
def test_last_odd_tile_row(K, m):
    _check(K, m, 2049)


@pytest.mark.parametrize("K", KS)
@pytest.mark.parametrize("tiles_out", [2, 148, 149, 296, 297, 444, 445])
@pytest.mark.parametrize("m,tiles_in", [(1, 16), (1, 17), (2, 16), (2, 17), (3, 5)])
def test_both_sides_of_every_switch(K, m, tiles_in, tiles_out):
    _check(K, m, tiles_out, tiles_in)


def _check(K, m, tiles_out, tiles_in=5):
    from trellis_b200 import qtip as q
    g = torch.Generator(device="cuda").manual_seed(K * 10 + m)
    packed = torch.randint(-2 ** 31, 2 ** 31, (tiles_out * tiles_in, 8 * K), dtype=torch.int64, generator=g, device="cuda").to(torch.int32)
    x = torch.randn(m, 16 * tiles_in, generator=g, device="cuda")
    y = q.decode_matvec(packed, 16 * tiles_out, 16 * tiles_in, K, "mcg", x)
    zq = q.from_tiles(q.decode_packed(packed, K, "mcg"), 16 * tiles_out, 16 * tiles_in).double()
    want = x.double() @ zq.t()
    assert y.shape == want.shape
    # at most 272 products in 32 partial sums: a few roundings each, 2e-6 of the norm as for the single-row form
    assert float(((y.double() - want).norm(dim=1) / want.norm(dim=1)).max()) < 2e-6
    assert float((y.double() - want)[:, -32:].abs().max()) < 2e-5 * float(want.abs().max())
