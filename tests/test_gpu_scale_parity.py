"""Parity at the sizes the benchmark runs.

(i)   GQA flash attention (`gqa_fmha_kernel<256,256>`) at M = 8192, 16 query / 2 KV heads, gated, partial rotary, FP8
      paged cache: one 8192-token call and a 4096 + 4096 two-chunk call, against the fp32 oracle on sampled query rows of
      the first, a middle and the last query tile; plus 20 differently seeded runs to flush data-dependent hangs
      (tests/test_attn_verify.py:197 of the reference accepts cos > 0.999).
(ii)  Gated DeltaNet at M = 8192 (128 chunks of 64) against `oracle.attention.gdn_layer_prefill` — output AND the carried
      fp32 state.
(iii) Grouped expert GEMMs at the expert geometries of every BASELINE config: DeepSeek-V2-Lite (H2048 I1408 E64 k6),
      Qwen3-235B (H4096 I1536 E128 k8), Qwen3.5-35B (H2048 I512 E256 k8) and Qwen3-Coder-Next (H2048 I512 E512 k10), INT4
      and INT8, 256 sampled tokens each against the oracle (reference tolerance precedent: tests/test_gpu_prefill.py:215-217).
(iv)  Router at 8192 x 512: every row whose ids differ from the oracle must be a near-tie row (k / k+1 logit gap, or a gap
      inside the top-k, below 1e-5); the near-tie rate is printed.
"""
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import attention as A, moe as omoe, router  # noqa: E402
from oracle.bf16 import f32_to_bf16_bits  # noqa: E402


# ------------------------------------------------------------------------------------------------ (i) GQA @ 8192

def _gqa_setup(nh, nkv, d, rot, gated, H, seed):
    torch.manual_seed(seed)
    bf = torch.bfloat16
    w = dict(q_proj=(torch.randn(nh * d * (2 if gated else 1), H) * 0.08).to(bf), k_proj=(torch.randn(nkv * d, H) * 0.08).to(bf),
             v_proj=(torch.randn(nkv * d, H) * 0.08).to(bf), o_proj=(torch.randn(H, nh * d) * 0.05).to(bf),
             q_norm=(1 + 0.1 * torch.randn(d)).to(bf), k_norm=(1 + 0.1 * torch.randn(d)).to(bf))
    cfg = types.SimpleNamespace(hidden_size=H, num_attention_heads=nh, num_key_value_heads=nkv, gqa_head_dim=d,
                                rotary_dim=rot, rope_theta=10000000.0, rms_norm_eps=1e-6)
    ocfg = dict(nh=nh, nkv=nkv, d=d, rotary_dim=rot, theta=10000000.0, eps=1e-6)
    return w, cfg, ocfg


def _sample_rows(M, q0=0):
    """Rows from the first, a middle and the last 128-row query tile (and the tile boundaries)."""
    rows = list(range(0, 48)) + list(range(120, 136)) + list(range(M // 2 - 24, M // 2 + 24)) + list(range(M - 64, M))
    return torch.tensor(sorted(set(r for r in rows if 0 <= r < M)), dtype=torch.long)


def _close(got, want, ulps, cos_min):
    err = (got - want).abs().max().item()
    assert err <= ulps * 2 ** -8 * want.abs().max().item(), (err, want.abs().max().item())
    cos = torch.nn.functional.cosine_similarity(got.reshape(1, -1), want.reshape(1, -1)).item()
    assert cos > cos_min, cos


@pytest.mark.parametrize("chunks", [(8192,), (4096, 4096)])
def test_gqa_fmha_at_8192_tokens_qcn_heads(chunks):
    from krasis_b200.attention import GQAAttention, PagedKVCache, SequenceKVState
    nh, nkv, d, rot, H = 16, 2, 256, 64, 512
    M = sum(chunks)
    w, cfg, ocfg = _gqa_setup(nh, nkv, d, rot, True, H, seed=77)
    x = torch.randn(M, H).to(torch.bfloat16)
    pos = torch.arange(M)
    att = GQAAttention(cfg, 0, w, "cuda:0", max_tokens=max(chunks))
    cache = PagedKVCache(1, nkv, d, "cuda:0", max_pages=M // 16 + 2)
    cache._free = [int(p) for p in np.random.default_rng(1).permutation(M // 16 + 2)]
    st = SequenceKVState(cache)
    got, start = [], 0
    for c in chunks:
        got.append(att.forward(x[start:start + c].cuda(), pos[start:start + c], cache, st, 0, c))
        st.advance(c)
        start += c
    torch.cuda.synchronize()
    kc = vc = None
    start = 0
    for c, g in zip(chunks, got):
        rows = _sample_rows(c)
        want, kc, vc = A.gqa_layer_prefill(x[start:start + c], w, ocfg, pos[start:start + c], kc, vc, rows=rows)
        _close(g.float().cpu()[rows], want.float(), ulps=4, cos_min=0.9995)
        start += c


def test_gqa_fmha_8192_twenty_seeds_complete_and_agree():
    """The lazy-rescale / double-buffered-P path is data dependent: run 20 different inputs (any hang trips the pytest
    timeout), check finiteness and run-to-run determinism on each."""
    from krasis_b200.attention import GQAAttention, PagedKVCache, SequenceKVState
    nh, nkv, d, rot, H, M = 16, 2, 256, 64, 256, 8192
    w, cfg, _ = _gqa_setup(nh, nkv, d, rot, True, H, seed=5)
    att = GQAAttention(cfg, 0, w, "cuda:0", max_tokens=M)
    cache = PagedKVCache(1, nkv, d, "cuda:0", max_pages=M // 16 + 1)
    pos = torch.arange(M)
    for seed in range(20):
        g = torch.Generator(device="cuda").manual_seed(100 + seed)
        scale = [0.3, 1.0, 4.0, 16.0][seed % 4]                 # wide logit ranges exercise the rescale branch
        x = (torch.randn(M, H, device="cuda", generator=g) * scale).to(torch.bfloat16)
        outs = []
        for _ in range(2):
            st = SequenceKVState(cache)
            outs.append(att.forward(x, pos, cache, st, 0, M))
            st.advance(M)
            st.free()
        torch.cuda.synchronize()
        assert torch.isfinite(outs[0].float()).all()
        assert torch.equal(outs[0], outs[1])


# ------------------------------------------------------------------------------------------------ (ii) GDN @ 8192

def test_gdn_at_8192_tokens_against_oracle():
    from krasis_b200.attention import GatedDeltaNetAttention
    torch.manual_seed(9)
    nk, nv, dk, dv, H, K, M = 4, 8, 128, 128, 256, 4, 8192
    kd, vd = nk * dk, nv * dv
    bf = torch.bfloat16
    w = dict(in_proj_qkvz=(torch.randn(2 * kd + 2 * vd, H) * 0.15).to(bf), in_proj_ba=(torch.randn(2 * nv, H) * 0.15).to(bf),
             out_proj=(torch.randn(H, vd) * 0.05).to(bf), conv1d_weight=(torch.randn(2 * kd + vd, 1, K) * 0.5).to(bf),
             A_log=(torch.randn(nv) * 0.5 - 1.0).to(bf), dt_bias=(torch.randn(nv) * 0.5).to(bf),
             norm_weight=(1 + 0.1 * torch.randn(dv)).to(bf))
    cfg = types.SimpleNamespace(hidden_size=H, linear_num_key_heads=nk, linear_num_value_heads=nv, linear_key_head_dim=dk,
                                linear_value_head_dim=dv, linear_conv_kernel_dim=K, rms_norm_eps=1e-6)
    x = torch.randn(M, H).to(bf)
    want, conv_o, st_o = A.gdn_layer_prefill(x, w, dict(nk=nk, nv=nv, dk=dk, dv=dv, eps=1e-6))
    lay = GatedDeltaNetAttention(cfg, 0, w, "cuda:0", max_tokens=M)
    got = lay.forward(x.cuda(), is_decode=False).float().cpu()
    conv, rec = lay.state()
    co = conv_o.float().numpy()
    assert np.abs(conv - co).max() <= 2 ** -7 * np.abs(co).max()
    # state after 128 chunks: same criterion as the short tests (BF16 inputs of the recurrence may flip by one ulp upstream)
    assert np.abs(rec - st_o.numpy()).max() < 5e-3 * max(1.0, st_o.abs().max().item())
    _close(got, want.float(), ulps=6, cos_min=0.9995)
    # the tail of the sequence is what carries 128 chunks of state: check it on its own
    _close(got[-512:], want.float()[-512:], ulps=6, cos_min=0.9995)


# ------------------------------------------------------------------------------------------------ (iii) expert geometries

GEOMETRIES = [("v2lite", 2048, 1408, 64, 6, 2048), ("q235b", 4096, 1536, 128, 8, 2048),
              ("qwen35", 2048, 512, 256, 8, 4096), ("qcn", 2048, 512, 512, 10, 8192)]


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("name,H,I,E,k,M", GEOMETRIES)
def test_moe_forward_at_baseline_geometries(name, H, I, E, k, M, bits):
    """Random weights in the reference QUANTISER's layout generated on the device, re-tiled by kb2_load_experts_dev;
    256 sampled tokens are routed inside a 12-expert subset (so the oracle only dequantises those), every other token is
    routed uniformly over all E experts — the kernels see the full geometry and a realistic load."""
    from krasis_b200 import KrasisEngine
    n_s, sub = 256, 12
    g = torch.Generator(device="cuda").manual_seed(H + I + E + bits)
    eng = KrasisEngine(hidden_size=H, moe_intermediate_size=I, n_routed_experts=E, num_experts_per_tok=k,
                       num_moe_layers=1, num_bits=bits, max_tokens=M)

    def rq(*shape):
        if bits == 4:
            return torch.randint(-2 ** 31, 2 ** 31 - 1, shape[:-1] + (shape[-1] // 8,), dtype=torch.int64, device="cuda", generator=g).to(torch.int32)
        return torch.randint(-128, 128, shape, dtype=torch.int64, device="cuda", generator=g).to(torch.int8)

    def rs(*shape):   # bf16 scales: |w| ~ 0.02 either way
        lo = 0.002 if bits == 4 else 0.0002
        return ((torch.rand(shape, device="cuda", generator=g) * 2 * lo + lo).to(torch.bfloat16)).view(torch.int16)

    w13_q, w13_s, w2_q, w2_s = rq(E, 2 * I, H), rs(E, 2 * I, H // 128), rq(E, H, I), rs(E, H, I // 128)
    eng.load_quantized_layer_dev(0, w13_q, w13_s, w2_q, w2_s)
    rng = np.random.default_rng(E + k)
    subset = np.sort(rng.choice(E, sub, replace=False))
    ids = np.stack([rng.choice(E, k, replace=False) for _ in range(M)]).astype(np.int32)
    sample = np.sort(rng.choice(M, n_s, replace=False))
    ids[sample] = np.stack([rng.choice(subset, k, replace=False) for _ in range(n_s)])
    wts = rng.dirichlet(np.ones(k), M).astype(np.float32)
    x = torch.randn(M, H, device="cuda", generator=g)
    x = (x / x.pow(2).mean(-1, keepdim=True).sqrt()).to(torch.bfloat16)
    out = eng.moe_forward(0, x, torch.from_numpy(ids).cuda(), torch.from_numpy(wts).cuda(), routed_only=True)
    torch.cuda.synchronize()
    counts = eng.last_expert_counts()
    assert np.array_equal(counts, np.bincount(ids.reshape(-1), minlength=E))
    # oracle on the sampled tokens: only the subset's experts are pulled to the host
    qdt = np.uint32 if bits == 4 else np.int8
    z13q = np.zeros((E,) + tuple(w13_q.shape[1:]), qdt); z13s = np.zeros((E, 2 * I, H // 128), np.uint16)
    z2q = np.zeros((E,) + tuple(w2_q.shape[1:]), qdt); z2s = np.zeros((E, H, I // 128), np.uint16)
    for e in subset:
        z13q[e] = w13_q[e].cpu().numpy().view(qdt); z13s[e] = w13_s[e].cpu().numpy().view(np.uint16)
        z2q[e] = w2_q[e].cpu().numpy().view(qdt); z2s[e] = w2_s[e].cpu().numpy().view(np.uint16)
    layer = omoe.Int4Layer(z13q, z13s, z2q, z2s, bits=bits)
    want = omoe.moe_forward_gpu_path(layer, x.float().cpu().numpy()[sample], ids[sample], wts[sample])
    got = out.float().cpu().numpy()[sample].astype(np.float64)
    rowmax = np.abs(want).max(axis=1, keepdims=True)
    assert (np.abs(got - want) <= 2 * rowmax * 2.0 ** -8 + 1e-30).all(), np.abs(got - want).max()
    cos = (got * want).sum() / (np.linalg.norm(got) * np.linalg.norm(want))
    assert cos >= 0.9999, cos
    out2 = eng.moe_forward(0, x, torch.from_numpy(ids).cuda(), torch.from_numpy(wts).cuda(), routed_only=True)
    assert torch.equal(out, out2)                                      # run-to-run determinism at full load
    eng.close()


# ------------------------------------------------------------------------------------------------ (iv) router @ 8192 x 512

@pytest.mark.parametrize("E,k,H", [(512, 10, 2048), (256, 8, 2048), (128, 8, 4096), (64, 6, 2048)])
def test_router_mismatches_are_near_ties_at_benchmark_size(E, k, H):
    from krasis_b200 import KrasisEngine
    M = 8192
    g = torch.Generator(device="cuda").manual_seed(E)
    x = torch.randn(M, H, device="cuda", generator=g)
    x = (x / x.pow(2).mean(-1, keepdim=True).sqrt()).to(torch.bfloat16)
    gate = (torch.randn(E, H, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    eng = KrasisEngine(hidden_size=H, moe_intermediate_size=512, n_routed_experts=E, num_experts_per_tok=k,
                       num_moe_layers=1, max_tokens=M, norm_topk_prob=True)
    eng.set_routing_weights(0, gate)
    ids, w = eng.compute_routing(0, x)
    lg = router.router_logits(x.float().cpu().numpy(), gate.float().cpu().numpy())
    ids_o, w_o = router.route_from_logits(lg, k, norm_topk_prob=True)
    gap = router.min_topk_gap(lg, k)
    near = gap < 1e-5
    differ = (ids.cpu().numpy() != ids_o).any(axis=1)
    print(f"router {M}x{E} top-{k}: near-tie rows {near.mean():.4%}, rows with different ids {differ.mean():.4%}")
    assert not (differ & ~near).any(), "a row away from every near-tie has different top-k ids"
    assert near.mean() < 0.02
    ok = ~near
    rel = np.abs(w.cpu().numpy()[ok] - w_o[ok]) / w_o[ok]
    assert rel.max() < 3e-5
    eng.close()


# ------------------------------------------------------------------------------------------------ tcgen05 scan vs mma.sync scan

@pytest.mark.parametrize("M", [200, 1024, 3000])
def test_gdn_tcgen05_scan_matches_the_mma_sync_scan(M, monkeypatch):
    """Same layer, same inputs, two state carries: the tcgen05 chunk scan (BF16 hi/lo pairs, fp32 accumulate) against the
    3xTF32 mma.sync scan kept for other head sizes.  Both are fp32-grade: the carried state must agree to 1e-4 relative,
    the BF16 outputs to one BF16 ulp of the output maximum's binade (2^-7 relative; rare rounding flips)."""
    from krasis_b200.attention import GatedDeltaNetAttention
    torch.manual_seed(21)
    nk, nv, dk, dv, H, K = 2, 4, 128, 128, 256, 4
    kd, vd = nk * dk, nv * dv
    bf = torch.bfloat16
    w = dict(in_proj_qkvz=(torch.randn(2 * kd + 2 * vd, H) * 0.15).to(bf), in_proj_ba=(torch.randn(2 * nv, H) * 0.15).to(bf),
             out_proj=(torch.randn(H, vd) * 0.05).to(bf), conv1d_weight=(torch.randn(2 * kd + vd, 1, K) * 0.5).to(bf),
             A_log=(torch.randn(nv) * 0.5).to(bf), dt_bias=(torch.randn(nv) * 0.5).to(bf),
             norm_weight=(1 + 0.1 * torch.randn(dv)).to(bf))
    cfg = types.SimpleNamespace(hidden_size=H, linear_num_key_heads=nk, linear_num_value_heads=nv, linear_key_head_dim=dk,
                                linear_value_head_dim=dv, linear_conv_kernel_dim=K, rms_norm_eps=1e-6)
    x1, x2 = torch.randn(M, H).to(bf).cuda(), torch.randn(M // 2 + 3, H).to(bf).cuda()
    res = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("KB2_GDN_LEGACY", mode)
        lay = GatedDeltaNetAttention(cfg, 0, w, "cuda:0", max_tokens=M)
        y1 = lay.forward(x1, is_decode=False).float().cpu()
        y2 = lay.forward(x2, is_decode=False).float().cpu()          # state carried into a second call
        _, rec = lay.state()
        res[mode] = (y1, y2, rec)
    for a, b in zip(res["0"][:2], res["1"][:2]):
        assert (a - b).abs().max().item() <= 2 ** -7 * b.abs().max().item()          # one BF16 ulp at the top binade
        assert (a == b).float().mean().item() > 0.95
    assert np.abs(res["0"][2] - res["1"][2]).max() <= 1e-4 * np.abs(res["1"][2]).max()


@pytest.mark.parametrize("M", [200, 1500, 4100])
def test_gdn_tcgen05_prepare_matches_the_mma_sync_prepare(M, monkeypatch):
    """tcgen05 chunk-prepare (explicit T = (I - A)^-1, BF16 hi/lo pairs of T times exact BF16 v / k) against the mma.sync
    prepare (blocked forward substitution on the right-hand sides), both feeding the same tcgen05 scan: fp32-grade both,
    so the carried state agrees to 1e-4 relative and the BF16 outputs to one ulp of the maximum."""
    from krasis_b200.attention import GatedDeltaNetAttention
    torch.manual_seed(22)
    nk, nv, dk, dv, H, K = 2, 4, 128, 128, 256, 4
    kd, vd = nk * dk, nv * dv
    bf = torch.bfloat16
    w = dict(in_proj_qkvz=(torch.randn(2 * kd + 2 * vd, H) * 0.15).to(bf), in_proj_ba=(torch.randn(2 * nv, H) * 0.15).to(bf),
             out_proj=(torch.randn(H, vd) * 0.05).to(bf), conv1d_weight=(torch.randn(2 * kd + vd, 1, K) * 0.5).to(bf),
             A_log=(torch.randn(nv) * 0.5).to(bf), dt_bias=(torch.randn(nv) * 0.5).to(bf),
             norm_weight=(1 + 0.1 * torch.randn(dv)).to(bf))
    cfg = types.SimpleNamespace(hidden_size=H, linear_num_key_heads=nk, linear_num_value_heads=nv, linear_key_head_dim=dk,
                                linear_value_head_dim=dv, linear_conv_kernel_dim=K, rms_norm_eps=1e-6)
    x1, x2 = torch.randn(M, H).to(bf).cuda(), torch.randn(M // 2 + 3, H).to(bf).cuda()
    res = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("KB2_GDN_PREPARE_MMA_SYNC", mode)
        lay = GatedDeltaNetAttention(cfg, 0, w, "cuda:0", max_tokens=M)
        y1 = lay.forward(x1, is_decode=False).float().cpu()
        y2 = lay.forward(x2, is_decode=False).float().cpu()
        _, rec = lay.state()
        res[mode] = (y1, y2, rec)
    for a, b in zip(res["0"][:2], res["1"][:2]):
        assert torch.isfinite(a).all()
        assert (a - b).abs().max().item() <= 2 ** -7 * b.abs().max().item()          # one BF16 ulp at the top binade
        assert (a == b).float().mean().item() > 0.95
    assert np.abs(res["0"][2] - res["1"][2]).max() <= 1e-4 * np.abs(res["1"][2]).max()
