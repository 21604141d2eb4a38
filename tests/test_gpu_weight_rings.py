"""Routed experts whose weights come from HBM, several K blocks of copies on their way and ending in any order: the bits of the same step on weights
that lie in L2."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import gguf_blocks as G, moe as omoe  # noqa: E402

TYPES = {"Q4_K": G.GGML_Q4_K, "Q8_0": G.GGML_Q8_0, "Q6_K": G.GGML_Q6_K}


# 50 and 500 rows per expert: wide chunks, one item per CTA and several; 6: short chunks
@pytest.mark.parametrize("gu,dn", [("Q4_K", "Q8_0"), ("Q4_K", "Q4_K"), ("Q8_0", "Q4_K"), ("Q6_K", "Q6_K")])
def test_cold_weights(gu, dn):
    from krasis_b200 import KrasisEngine
    E, H, I, k = 32, 1024, 512, 4
    rng = np.random.default_rng(0)
    lay = omoe.make_gguf_layer(rng, E, H, I, gate_up_type=TYPES[gu], down_type=TYPES[dn])
    eng = KrasisEngine(hidden_size=H, moe_intermediate_size=I, n_routed_experts=E, num_experts_per_tok=k, num_moe_layers=1, max_tokens=4000,
                       gguf_gate_up_type=gu, gguf_down_type=dn)
    eng.load_gguf_layer(0, lay.gate, lay.up, lay.down)
    spoil = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")          # more than L2 holds
    g = torch.Generator(device="cuda").manual_seed(1)
    for M in (48, 400, 4000):
        x = torch.randn(M, H, device="cuda", generator=g).bfloat16()
        ids = torch.rand(M, E, device="cuda", generator=g).argsort(1)[:, :k].int().contiguous()
        w = torch.rand(M, k, device="cuda", generator=g)
        want = eng.moe_forward(0, x, ids, w, routed_only=True)
        for _ in range(10):
            spoil.zero_()
            assert torch.equal(eng.moe_forward(0, x, ids, w, routed_only=True), want)
