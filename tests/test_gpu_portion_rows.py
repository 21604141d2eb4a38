"""The operands of a portion's attention in one launch, against torch's gathers and conversions, and the attention's bfloat16 rows."""
import pytest
import torch

from krasis_b200 import seqops as ops

pytestmark = pytest.mark.gpu


# first rows in the middle of a page, portions of one token, widths of one 16-byte group, rows of the projection that start off 16 bytes
@pytest.mark.parametrize("wa,wb,nq,ld", [(256, 256, 2048, 2560), (512, 64, 3072, 3648), (8, 8, 8, 11), (128, 256, 128, 130)])
@pytest.mark.parametrize("start,n,first", [(0, 1, 0), (70, 130, 3), (64, 64, 64), (200, 17, 137)])
def test_portion_rows(wa, wb, nq, ld, start, n, first):
    g = torch.Generator(device="cuda").manual_seed(wa + n)
    page, total = 64, start + n
    pages = torch.randperm(9, generator=torch.Generator().manual_seed(n))[:(total + page - 1) // page].tolist()
    ca, cb = torch.randn(9, page, wa, device="cuda", generator=g).bfloat16(), torch.randn(9, page, wb, device="cuda", generator=g).bfloat16()
    proj = torch.randn(n + 2, ld, device="cuda", generator=g)
    tb = ops.StepTables([([0], 5, 1, [8]), ([0] * n, start, 0, pages)], "cuda")
    a, b, q = ops.portion_rows(tb, 1, first, ca, wa, cb, wb, page, proj, 1, n, nq)
    rows = torch.tensor([pages[j // page] * page + j % page for j in range(first, total)], device="cuda")
    assert torch.equal(a, ca.view(-1, wa)[rows]) and torch.equal(b, cb.view(-1, wb)[rows]) and torch.equal(q, proj[1:1 + n, :nq].bfloat16())


@pytest.mark.parametrize("n,start,window,sink", [(128, 0, 0, False), (131, 77, 100, True), (300, 1, 0, True)])
def test_rows_rounded_by_the_attention(n, start, window, sink):
    """Heads without a norm, gate or maps are written in bfloat16 by the attention itself: the same bits as fp32 rows finished in a pass of
    their own (coefficients of one, which that pass multiplies by)."""
    from krasis_b200.mixers import MultiMapAttention
    H, G, d, W = 4, 2, 128, 256
    g = torch.Generator().manual_seed(n)
    w = {"q": torch.randn(H * d, W, generator=g), "k": torch.randn(G * d, W, generator=g), "v": torch.randn(G * d, W, generator=g),
         "o": torch.randn(W, H * d, generator=g)}
    w = {k: v * W ** -0.5 for k, v in w.items()}
    if sink:
        w["sink"] = torch.randn(H, generator=g)
    pages = [3, 0, 5, 1, 4, 2, 6][:(start + n + 63) // 64]
    tb = ops.StepTables([([0] * n, start, 0, pages)], "cuda")
    h = torch.randn(n, W, generator=g).bfloat16().cuda()
    kc, vc = (torch.randn(7, 64, G * d, generator=g).bfloat16().cuda() for _ in range(2))
    out = []
    for coef in (None, [1.0]):
        m = MultiMapAttention(w, H, G, 1, d, d, d ** -0.5, 1e-5, torch.bfloat16, "cuda", window=window or None, map_coef=coef)
        out.append(m.forward(h, tb, kc.clone(), vc.clone(), 64))
    assert torch.equal(out[0], out[1]) and torch.isfinite(out[0]).all()
