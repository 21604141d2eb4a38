"""Token tiles of the DeltaNet preparation, sixteen rows in groups of four and a remainder: a prompt in one call against the same prompt in parts (history from
the convolution state)."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,cuts", [(2049, (2048,)), (2100, (15, 16, 17, 64)), (2113, (1, 1024, 2112))])
def test_one_call_and_parts_agree(M, cuts):
    from krasis_b200.attention import GatedDeltaNetAttention
    torch.manual_seed(M)
    nk, nv, d, H, K = 4, 8, 128, 256, 4
    kd, vd = nk * d, nv * d
    bf = torch.bfloat16
    w = dict(in_proj_qkvz=(torch.randn(2 * kd + 2 * vd, H) * 0.15).to(bf), in_proj_ba=(torch.randn(2 * nv, H) * 0.15).to(bf),
             out_proj=(torch.randn(H, vd) * 0.05).to(bf), conv1d_weight=(torch.randn(2 * kd + vd, 1, K) * 0.5).to(bf),
             A_log=(torch.randn(nv) * 0.5).to(bf), dt_bias=(torch.randn(nv) * 0.5).to(bf), norm_weight=(1 + 0.1 * torch.randn(d)).to(bf))
    cfg = types.SimpleNamespace(hidden_size=H, linear_num_key_heads=nk, linear_num_value_heads=nv, linear_key_head_dim=d,
                                linear_value_head_dim=d, linear_conv_kernel_dim=K, rms_norm_eps=1e-6)
    lay = GatedDeltaNetAttention(cfg, 0, w, "cuda:0", max_tokens=M)
    x = torch.randn(M, H).to(bf).cuda()
    whole = lay.forward(x, is_decode=False).float()
    conv, rec = lay.state()
    lay.reset_state()
    edges = [0, *cuts, M]
    parts = torch.cat([lay.forward(x[a:b].contiguous(), is_decode=False).float() for a, b in zip(edges, edges[1:])])
    conv2, rec2 = lay.state()
    # projections of different row counts sum in another order, and a cut that is no multiple of 64 moves the recurrence's chunks: a bf16
    # neighbour per stage (projection, convolution, read-out, output) of the row's largest value
    assert abs(conv - conv2).max() <= 2 ** -7 * abs(conv).max()
    assert abs(rec - rec2).max() <= 5e-3 * max(1.0, abs(rec).max())
    assert (whole - parts).abs().max() <= 3 * 2 ** -7 * whole.abs().max()


@pytest.mark.parametrize("M,cuts", [(20, (1, 3, 6, 10, 15)), (31, (16, 23)), (45, (13, 14, 27, 36))])
def test_remainders_of_a_tile(M, cuts):
    """Calls of 1 to 16 tokens, and 17 and more: every number of rows in the last group of four."""
    test_one_call_and_parts_agree(M, cuts)
