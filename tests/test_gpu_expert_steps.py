"""Short steps of routed experts: short chunks, one-launch binning and narrow router tiles against the forms that long steps take."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import moe as omoe, router  # noqa: E402
from oracle.bf16 import f32_to_bf16_bits, round_bf16  # noqa: E402
from tests.test_gpu_moe import bf16_t, make_engine  # noqa: E402

GGUF = {"Q8_0": ("Q8_0", "Q8_0"), "Q4_K": ("Q4_K", "Q6_K")}


def _engine(fmt, rng, E, H, I, k, M):
    if fmt in (4, 8):
        return make_engine(omoe.make_int_layer(rng, E, H, I, bits=fmt), k, M, num_bits=fmt)
    from krasis_b200 import KrasisEngine
    from oracle import gguf_blocks as G
    T = {"Q4_K": G.GGML_Q4_K, "Q8_0": G.GGML_Q8_0, "Q6_K": G.GGML_Q6_K}
    gu, dn = GGUF[fmt]
    lay = omoe.make_gguf_layer(rng, E, H, I, gate_up_type=T[gu], down_type=T[dn])
    eng = KrasisEngine(hidden_size=H, moe_intermediate_size=I, n_routed_experts=E, num_experts_per_tok=k, num_moe_layers=1,
                       max_tokens=M, gguf_gate_up_type=gu, gguf_down_type=dn)
    eng.load_gguf_layer(0, lay.gate, lay.up, lay.down)
    return eng


@pytest.mark.parametrize("fmt", [4, 8, "Q8_0", "Q4_K"])
@pytest.mark.parametrize("skew", [0.0, 4.0])
def test_rows_do_not_depend_on_the_length_of_the_step(fmt, skew):
    """A row's result is one sum in a fixed order whatever chunk holds it: the first rows of a long step (mean 250 rows per expert: wide chunks,
    three-launch binning) come out bit for bit in steps that take short chunks and the one-launch binning.  With the skew expert 0 gets nearly every
    row, so its run is cut into several short chunks."""
    rng = np.random.default_rng(5)
    E, H, I, k, M = 16, 512, 256, 2, 2100                      # 4200 entries: past the one-launch binning
    eng = _engine(fmt, rng, E, H, I, k, M)
    x = round_bf16(rng.normal(0, 1, (M, H)).astype(np.float32))
    lg = rng.normal(0, 1, (M, E)).astype(np.float32)
    lg[:, 0] += skew
    ids, w = router.route_from_logits(lg, k, norm_topk_prob=True)
    ids[1] = -1                                                # a row without experts, one with a single one
    ids[2, 0] = -1
    tx, ti, tw = bf16_t(x), torch.from_numpy(ids).cuda(), torch.from_numpy(w).cuda()
    want = eng.moe_forward(0, tx, ti, tw, routed_only=True)
    for m in (1, 3, 16, 17, 64, 65, 129, 384, 385, 512, 513, 2048):      # 48 and 64 rows per expert, the last short steps; 2048: 4096 entries
        got = eng.moe_forward(0, tx[:m], ti[:m], tw[:m], routed_only=True)
        assert torch.equal(got, want[:m]), m
        assert np.array_equal(eng.last_expert_counts(), np.bincount(ids[:m][ids[:m] >= 0], minlength=E)), m
    assert (want[1] == 0).all() and torch.isfinite(want.float()).all()


@pytest.mark.parametrize("E,k", [(33, 5), (64, 8), (100, 32), (200, 8), (512, 10), (1000, 32)])
@pytest.mark.parametrize("scoring", ["softmax", "sigmoid"])
def test_choice_among_ties_is_by_index(E, k, scoring):
    """Logits from a handful of values: the choice is the stable descending order, the weights those of the chosen scores."""
    from krasis_b200 import KrasisEngine
    rng = np.random.default_rng(E + k)
    H, M = 256, 40
    gate = np.zeros((E, H), np.float32)
    gate[:, :M] = rng.choice([-1.0, -0.5, -0.0, 0.0, 0.25, 1.5], (E, M))
    hid = np.zeros((M, H), np.float32)
    hid[np.arange(M), np.arange(M)] = 1.0                      # logits of token m = column m of the gate, exactly
    eng = KrasisEngine(hidden_size=H, moe_intermediate_size=128, n_routed_experts=E, num_experts_per_tok=k, num_moe_layers=1, max_tokens=M,
                       scoring_func=scoring, norm_topk_prob=False)
    eng.set_routing_weights(0, f32_to_bf16_bits(gate))
    ids, w = eng.compute_routing(0, bf16_t(hid))
    lg = gate[:, :M].T.astype(np.float64)
    want = np.argsort(-lg, axis=1, kind="stable")[:, :k]
    assert np.array_equal(ids.cpu().numpy(), want)
    score = np.exp(lg) / np.exp(lg).sum(1, keepdims=True) if scoring == "softmax" else 1 / (1 + np.exp(-lg))
    assert np.allclose(w.cpu().numpy(), np.take_along_axis(score, want, 1), rtol=1e-5)      # a few fp32 roundings and expf's two ulp


@pytest.mark.parametrize("M", [1, 127, 129, 2304, 2305])
def test_router_tiles_agree(M):
    """512 experts: narrow tiles up to 18 x 8 of them, wide ones past that; the same choice and weights for the same rows."""
    from krasis_b200 import KrasisEngine
    rng = np.random.default_rng(3)
    E, H, k = 512, 1024, 10
    x = round_bf16(rng.normal(0, 1, (2500, H)).astype(np.float32))
    eng = KrasisEngine(hidden_size=H, moe_intermediate_size=128, n_routed_experts=E, num_experts_per_tok=k, num_moe_layers=1, max_tokens=2500,
                       norm_topk_prob=True)
    eng.set_routing_weights(0, f32_to_bf16_bits(round_bf16(rng.normal(0, 0.02, (E, H)).astype(np.float32))))
    tx = bf16_t(x)
    want_ids, want_w = eng.compute_routing(0, tx)
    ids, w = eng.compute_routing(0, tx[:M])
    assert torch.equal(ids, want_ids[:M]) and torch.equal(w, want_w[:M])
