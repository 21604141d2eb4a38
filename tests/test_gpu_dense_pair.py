"""Dense products on pairs of CTAs: the sums of the one-CTA tiles and of the few-row tiles, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _form(M, N, K):
    from krasis_b200 import capi
    return capi.load().kb2_linear_bf16_form(M, N, K, 0, None)


# rows around the pair's 256 and one CTA's 128, columns that end in the first or the second CTA's half of a tile, tiles of 96 to 256 columns, several rounds
PAIRS = [(2304, 576, 2048), (2500, 3648, 2048), (2113, 12352, 2048), (1024, 16384, 1024), (4096, 9216, 2048), (1500, 2048, 2048), (3333, 1040, 4096),
         (8192, 592, 2048), (4481, 1040, 4096)]


def test_these_run_on_pairs():
    """The form follows from estimates: without this a change of theirs could leave the pair kernel untested."""
    forms = {s: _form(*s) for s in PAIRS}
    assert all(f > 0 for f in forms.values()) and len(set(forms.values())) >= 5, forms


# and shapes of one K block or a few, which run on one CTA per tile
@pytest.mark.parametrize("M,N,K", PAIRS + [(2049, 16, 64), (2304, 272, 128), (2100, 2048, 192), (4481, 1040, 576), (8192, 528, 256), (2113, 12352, 320),
                                           (700, 16384, 256), (1500, 9216, 512)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_rows_equal_those_of_few(M, N, K, out_dtype):
    from krasis_b200.attention import linear
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    got = linear(x, w, out_dtype=out_dtype)
    want = x.double() @ w.double().T
    # one accumulator that cuts off what each instruction adds: 2^-23 of the terms' magnitudes for every 16 of K, and the rounding of the result
    room = 2.0 ** -23 * (K / 16) * (x.double().abs() @ w.double().abs().T) + (2.0 ** -8 * want.abs() if out_dtype == torch.bfloat16 else 0.0)
    assert ((got.double() - want).abs() <= room).all()
    if out_dtype == torch.bfloat16:                # 200 rows run on tiles of few rows (fp32 outputs of few rows are summed in chunks)
        for at in (0, 127, 255, M - 200):
            assert torch.equal(linear(x[at:at + 200].contiguous(), w, out_dtype=out_dtype), got[at:at + 200])


@pytest.mark.parametrize("M,H", [(2304, 576), (4610, 576)])
def test_rows_of_owners(M, H):
    """Output rows that go straight into the receive buffers of the ranks that own them, long steps on pairs of CTAs: two buffers on this GPU."""
    import types
    from krasis_b200 import attention as A
    nh, d = 16, 128
    assert _form(M, H, nh * d) > 0
    cfg = types.SimpleNamespace(hidden_size=H, num_attention_heads=nh, num_key_value_heads=2, gqa_head_dim=d, rotary_dim=64, rope_theta=10000.0,
                                rms_norm_eps=1e-6)
    g = torch.Generator(device="cuda").manual_seed(M)
    bf = lambda *s, sd=1.0: (torch.randn(*s, device="cuda", generator=g) * sd).bfloat16()  # noqa: E731
    w = dict(q_proj=bf(nh * d, H, sd=H ** -0.5), k_proj=bf(2 * d, H, sd=H ** -0.5), v_proj=bf(2 * d, H, sd=H ** -0.5), o_proj=bf(H, nh * d, sd=0.05),
             q_norm=bf(d) * 0.1 + 1, k_norm=bf(d) * 0.1 + 1)
    layer, cache = A.GQAAttention(cfg, 0, w, "cuda:0", max_tokens=M), A.PagedKVCache(1, 2, d, "cuda:0", M // 16 + 2)
    seq, x, pos = A.SequenceKVState(cache), bf(M, H), torch.arange(M, dtype=torch.int32, device="cuda")
    want = layer.forward(x, pos, cache, seq, 0, M)
    recv = [torch.zeros(M // 2, 2, H, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    layer.set_output_scatter([r.data_ptr() for r in recv], 1)
    layer.forward(x, pos, cache, seq, 0, M)
    layer.set_output_scatter(None)
    got = torch.cat(recv, 0)
    assert torch.equal(got[:, 1], want) and (got[:, 0] == 0).all() and want.float().norm() > 0
