"""Gated units that the product writes itself: the bits of the product into bfloat16 rows and the activation pass."""
import pytest
import torch

from krasis_b200 import mixers
from krasis_b200.mixers import GatedMLP, RoutedExperts

pytestmark = pytest.mark.gpu


# rows and columns around the tiles (64 columns of gate and of up to a tile), one and several CTAs along K, steps of 256 rows and more
@pytest.mark.parametrize("act,limit", [("silu", 0.0), ("gelu_tanh", 0.0), ("clamped_swish", 0.8)])
@pytest.mark.parametrize("M,F,W", [(9, 128, 64), (16, 144, 256), (77, 992, 2048), (129, 2096, 512), (255, 576, 4096), (256, 512, 2048), (300, 272, 7168)])
def test_gated_mlp(M, F, W, act, limit, monkeypatch):
    g = torch.Generator().manual_seed(M + F)
    w = {"gate": torch.randn(F, W, generator=g) * W ** -0.5, "up": torch.randn(F, W, generator=g) * W ** -0.5, "down": torch.randn(W, F, generator=g) * F ** -0.5}
    m = GatedMLP(w, torch.bfloat16, "cuda", act=act, limit=limit, alpha=1.7)
    h = torch.randn(M, W, generator=g).bfloat16().cuda()
    h[0, :3] = torch.tensor([float("inf"), float("nan"), -3e38])
    unit = mixers.lin_glu(h, m.w_gu, m.kind, m.limit, m.alpha)
    got = m.forward(h)
    monkeypatch.setattr(mixers, "lin_glu", lambda *a: None)
    assert torch.equal(got.view(torch.int32), m.forward(h).view(torch.int32))
    assert unit is not None or M >= 256
    z = (h[1:].double().cpu() @ torch.cat([w["gate"], w["up"]]).bfloat16().double().T).bfloat16().double()
    a, b = z[:, :F], z[:, F:]
    if act == "clamped_swish":
        a, b = a.clamp(max=limit), b.clamp(-limit, limit)
    want = {"silu": a * torch.sigmoid(a) * b, "gelu_tanh": torch.nn.functional.gelu(a, approximate="tanh") * b,
            "clamped_swish": a * torch.sigmoid(1.7 * a) * (b + 1)}[act]
    if unit is not None:          # both factors within a unit in the last place of bfloat16 (2^-8) of the rounded products, slopes below 1.13 and 1.7 * 0.8
        assert ((unit[1:].double().cpu() - want).abs() <= 2.0 ** -6 * ((1 + a.abs()) * (1 + b.abs()))).all()


# tiles of 16, 32, 48 and 64 rows; 24 experts leave runs empty; F of one to five tiles of 64 columns; one and several CTAs along K
@pytest.mark.parametrize("T,E,top,F,W", [(9, 24, 3, 128, 256), (40, 8, 4, 192, 512), (80, 8, 4, 64, 256), (100, 8, 4, 320, 512), (12, 2, 1, 64, 8192)])
@pytest.mark.parametrize("act", ["silu", "clamped_swish"])
def test_routed_experts(T, E, top, F, W, act):
    g = torch.Generator().manual_seed(T + F)
    w = {"router": torch.randn(E, W, generator=g) * W ** -0.5}
    for i in range(E):
        w.update({f"e{i}_gate": torch.randn(F, W, generator=g) * W ** -0.5, f"e{i}_up": torch.randn(F, W, generator=g) * W ** -0.5,
                  f"e{i}_down": torch.randn(W, F, generator=g) * F ** -0.5})
    m = RoutedExperts(w, E, 0, top, torch.bfloat16, "cuda", act=act, limit=0.9, alpha=1.7)
    h = torch.randn(T, W, generator=g).bfloat16().cuda()
    assert m._tile_rows(T * top) < 128
    ids = m.route(h)[0]
    got, pos = m._forward_tensor_core(h, ids, T * top, None)
    want, pos2 = m._forward_tensor_core(h, ids, T * top, torch.ones(T * top, device="cuda"))   # weights of one on the inputs: the product and the pass
    # the order within an expert's run may differ between two binnings
    assert torch.equal(got[pos.long()].view(torch.int32), want[pos2.long()].view(torch.int32))
