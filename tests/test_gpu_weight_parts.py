"""fp32 products whose weights need no low parts (a bf16 checkpoint in the fp32 mode): left out where they are zeros, with the same sums."""
import pytest
import torch

from krasis_b200 import mixers

pytestmark = pytest.mark.gpu


# K of one span of blocks, of several and a short one, and beyond 32 spans of four; columns that end inside a tile; one head and several
@pytest.mark.parametrize("M,N,K,G", [(9, 16, 128, 1), (77, 320, 576, 1), (130, 144, 8256, 1), (300, 256, 2304, 3), (33, 2048, 2048, 1)])
@pytest.mark.parametrize("where", ["first", "last", "everywhere"])
def test_zero_parts_left_out(M, N, K, G, where):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, G, K, device="cuda", generator=g)
    w = (torch.randn(G, N, K, device="cuda", generator=g) * K ** -0.5).bfloat16().float()
    out = torch.empty(M, G, N, device="cuda")
    assert mixers._lin_f32(x, w, out)
    want = torch.einsum("mgk,gnk->mgn", x.double(), w.double())
    room = 2.0 ** -21 * torch.einsum("mgk,gnk->mgn", x.double().abs(), w.double().abs())
    assert ((out.double() - want).abs() <= room).all()
    # one row of every tile of 128 gets numbers that need their low parts, at the span's first or last number or all along the row: the other rows
    # of its tile keep their sums bit for bit
    mixed, rows = w.clone(), list(range(0, N, 128)) if where != "last" else [min(n + 127, N - 1) for n in range(0, N, 128)]
    for r in rows:
        k = slice(None) if where == "everywhere" else 0 if where == "first" else min(255, K - 1)
        mixed[:, r, k] = torch.randn_like(mixed[:, r, k])
    got = torch.empty_like(out)
    assert mixers._lin_f32(x, mixed, got)
    others = [n for n in range(N) if n not in rows]
    assert torch.equal(got[:, :, others], out[:, :, others])
    want = torch.einsum("mgk,gnk->mgn", x.double(), mixed.double())
    room = 2.0 ** -21 * torch.einsum("mgk,gnk->mgn", x.double().abs(), mixed.double().abs())
    assert ((got.double() - want).abs() <= room).all()
