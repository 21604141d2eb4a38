"""The work a user of this framework has it do, as cases that can be timed and checked.

Two halves, as the framework has: the blocks of the MoE prefill models (routed experts, Gated DeltaNet, grouped-query and latent attention,
W8A8 shared expert) at the geometries of the presets in krasis_b200.model, and ragged-batch serving (feed-forward units, routed experts,
recurrent and attention mixers, whole steps through the scheduler) at the geometries of krasis_b200.bench_seq.  Every case goes through an
entry point that a program calls; `exact` restates it in float64 with plain torch.

  listed() / draw(rng)       the cases; prepare(case, seed) / run(state) one pass; work(case) what it cannot do without;
  tolerance(case)            how far another correct implementation may be off; exact(case, seed) the float64 result
"""
import math
import types

import torch

DEV = "cuda:0"
BF = torch.bfloat16
W = 2048                                     # width of every model of the benchmark and of three of the four presets

# expert geometries of the presets: experts, top-k, intermediate size, renormalised weights
EXPERTS = {"qcn": (512, 10, 512, True), "qwen35": (256, 8, 512, True), "v2lite": (64, 6, 1408, False)}
MAXT = 8192                                  # the prompt length the headline metric is quoted on


def listed():
    return [
        # ---- MoE prefill models
        # one whole prompt of the headline benchmark through a MoE layer (router, 512 INT4 experts, top 10)
        {"name": "experts_prompt", "kind": "experts", "model": "qcn", "bits": 4, "tokens": 8192},
        # a short question to the INT8 form of the smaller model: each expert gets a few dozen rows
        {"name": "experts_question_int8", "kind": "experts", "model": "v2lite", "bits": 8, "tokens": 389},
        # the smallest call: a few tokens, launches and weight streaming only
        {"name": "experts_few", "kind": "experts", "model": "qwen35", "bits": 4, "tokens": 3},
        # the linear-attention block of three layers out of four, a prompt of ragged length
        {"name": "deltanet_prompt", "kind": "deltanet", "tokens": 3333},
        # the gated full-attention block of every fourth layer: a second portion of a prompt on top of cached keys
        {"name": "gqa_portion", "kind": "gqa", "tokens": 2048, "past": 2500},
        # latent attention of the smaller model, a medium prompt
        {"name": "mla_prompt", "kind": "mla", "tokens": 1000, "past": 0},
        # ---- ragged-batch serving
        # dense feed-forward on a step of a few dozen tokens: the tail of a prompt beside decoded tokens
        {"name": "ffn_tail", "kind": "ffn", "tokens": 77, "dtype": "bfloat16", "act": "silu"},
        # the same unit in the fp32 mode of the trace runner
        {"name": "ffn_fp32", "kind": "ffn", "tokens": 512, "dtype": "float32", "act": "gelu_tanh"},
        # routed bf16 experts on a portion of a prompt
        {"name": "moe_portion", "kind": "moe", "tokens": 128, "dtype": "bfloat16"},
        # gated delta rule over a whole prompt of the serving benchmark
        {"name": "delta_prompt", "kind": "delta", "tokens": 4096, "dtype": "bfloat16"},
        # windowed attention on a mixed step: one portion of a prompt and three requests that decode
        {"name": "attention_mixed", "kind": "attention", "tokens": 512, "past": 700, "decoding": 3, "context": 2048, "window": 1024,
         "dtype": "bfloat16"},
        # whole model through the scheduler: short prompts are admitted, then every request decodes (captured steps)
        {"name": "serve_decode", "kind": "serve", "requests": 4, "prompt": 100, "decode": 16, "dtype": "bfloat16"},
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["experts", "experts", "deltanet", "gqa", "mla", "shared", "ffn", "ffn", "moe", "delta", "attention", "attention", "serve"])
    dtype = "float32" if rng.random() < 0.15 else "bfloat16"
    if kind == "experts":
        model = rng.choice(sorted(EXPERTS))
        # the routed width of a whole prompt is the largest listed case: the others stay below it
        return {"kind": kind, "model": model, "bits": rng.choice([4, 4, 8]), "tokens": _logint(rng, 1, 6000)}
    if kind == "deltanet":
        return {"kind": kind, "tokens": _logint(rng, 16, 3300)}
    if kind in ("gqa", "mla"):
        return {"kind": kind, "tokens": _logint(rng, 16, 2000), "past": rng.choice([0, 0, _logint(rng, 16, 2500)])}
    if kind == "shared":
        return {"kind": kind, "tokens": _logint(rng, 16, 8192)}
    if kind == "ffn":
        return {"kind": kind, "tokens": _logint(rng, 1, 4096 if dtype == "bfloat16" else 500), "dtype": dtype, "act": rng.choice(["silu", "gelu_tanh"])}
    if kind == "moe":
        return {"kind": kind, "tokens": _logint(rng, 1, 4096 if dtype == "bfloat16" else 100), "dtype": dtype}
    if kind == "delta":
        return {"kind": kind, "tokens": _logint(rng, 1, 4000), "dtype": dtype if rng.random() < 0.5 else "bfloat16"}
    if kind == "attention":
        return {"kind": kind, "tokens": _logint(rng, 16, 2048 if dtype == "bfloat16" else 256), "past": rng.choice([0, _logint(rng, 16, 2000)]),
                "decoding": rng.randint(0, 6), "context": _logint(rng, 64, 4000), "window": rng.choice([1024, 0]), "dtype": dtype}
    return {"kind": kind, "requests": rng.randint(1, 6), "prompt": _logint(rng, 4, 300), "decode": rng.randint(4, 20), "dtype": "bfloat16"}


# ------------------------------------------------------------------------------------------------ inputs

class Draws:
    """Tensors from the seed alone, on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 62))

    def n(self, *shape, sd=1.0, mean=0.0):
        return torch.randn(*shape, device=DEV, generator=self.g) * sd + mean

    def bf(self, *shape, sd=1.0, mean=0.0):
        return self.n(*shape, sd=sd, mean=mean).to(BF)

    def ints(self, lo, hi, *shape, dtype=torch.int64):
        return torch.randint(lo, hi, shape, device=DEV, generator=self.g, dtype=dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, device=DEV, generator=self.g) * (hi - lo) + lo


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else BF


def _in_experts(case, seed):
    """Router, hidden rows and one layer of quantised experts as the group quantiser emits them: q in [-7, 7] (INT4) or [-127, 127]."""
    E, k, I, _ = EXPERTS[case["model"]]
    d = Draws(seed)
    x, gate = d.bf(case["tokens"], W), d.bf(E, W, sd=W ** -0.5)
    out = {"x": x, "gate": gate}
    for name, rows, cols in (("w13", 2 * I, W), ("w2", W, I)):
        if case["bits"] == 4:
            words = torch.zeros(E, rows, cols // 8, dtype=torch.int64, device=DEV)
            for i in range(8):
                words |= d.ints(1, 16, E, rows, cols // 8) << (4 * i)
            out[name + "_q"] = torch.where(words >= 1 << 31, words - (1 << 32), words).to(torch.int32)
            top = 7.0
        else:
            out[name + "_q"] = d.ints(-127, 128, E, rows, cols, dtype=torch.int8)
            top = 127.0
        out[name + "_s"] = d.uniform(0.5, 1.5, E, rows, cols // 128).mul_(cols ** -0.5 * 1.7 / top).to(BF)
    return out


def _dequant(q, s, bits):
    """[rows, cols] float64 values of one expert's quantised matrix."""
    if bits == 4:
        q = ((q.unsqueeze(-1) >> (4 * torch.arange(8, device=q.device, dtype=torch.int32))) & 15).reshape(q.shape[0], -1) - 8
    return (q.double().view(q.shape[0], -1, 128) * s.double().unsqueeze(-1)).view(q.shape[0], -1)


DN = types.SimpleNamespace(hidden_size=W, linear_num_key_heads=16, linear_num_value_heads=32, linear_key_head_dim=128,
                           linear_value_head_dim=128, linear_conv_kernel_dim=4, rms_norm_eps=1e-6)


def _in_deltanet(case, seed):
    d, kd, vd = Draws(seed), 16 * 128, 32 * 128
    w = dict(in_proj_qkvz=d.bf(2 * kd + 2 * vd, W, sd=W ** -0.5), in_proj_ba=d.bf(64, W, sd=W ** -0.5), out_proj=d.bf(W, vd, sd=vd ** -0.5),
             conv1d_weight=d.bf(2 * kd + vd, 1, 4, sd=0.5), A_log=torch.log(d.uniform(1.0, 8.0, 32)).to(BF), dt_bias=d.bf(32, mean=-3.0),
             norm_weight=d.bf(128, sd=0.1, mean=1.0))
    return d.bf(case["tokens"], W), w


GQA = types.SimpleNamespace(hidden_size=W, num_attention_heads=16, num_key_value_heads=2, gqa_head_dim=256, rotary_dim=64,
                            rope_theta=10000000.0, rms_norm_eps=1e-6)


def _in_gqa(case, seed):
    d = Draws(seed)
    w = dict(q_proj=d.bf(2 * 16 * 256, W, sd=W ** -0.5), k_proj=d.bf(512, W, sd=W ** -0.5), v_proj=d.bf(512, W, sd=W ** -0.5),
             o_proj=d.bf(W, 4096, sd=4096 ** -0.5), q_norm=d.bf(256, sd=0.1, mean=1.0), k_norm=d.bf(256, sd=0.1, mean=1.0))
    kc, vc = (d.n(case["past"] + case["tokens"], 512).to(torch.float8_e4m3fn) for _ in range(2))
    return d.bf(case["tokens"], W), w, kc, vc


MLA_ROPE = {"beta_fast": 32, "beta_slow": 1, "factor": 40, "mscale": 0.707, "mscale_all_dim": 0.707, "original_max_position_embeddings": 4096}
MLA = types.SimpleNamespace(hidden_size=W, num_attention_heads=16, qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128,
                            kv_lora_rank=512, q_lora_rank=None, rope_theta=10000.0, rope_scaling=MLA_ROPE, rms_norm_eps=1e-6)


def _in_mla(case, seed):
    d = Draws(seed)
    w = dict(q_proj=d.bf(16 * 192, W, sd=W ** -0.5), kv_a_proj_with_mqa=d.bf(576, W, sd=W ** -0.5), kv_a_layernorm=d.bf(512, sd=0.1, mean=1.0),
             w_kc=d.bf(16, 128, 512, sd=512 ** -0.5), w_vc=d.bf(16, 128, 512, sd=512 ** -0.5), o_proj=d.bf(W, 2048, sd=W ** -0.5))
    total = case["past"] + case["tokens"]
    ckv, kpe = d.n(total, 512).to(torch.float8_e4m3fn), d.n(total, 64).to(torch.float8_e4m3fn)
    return d.bf(case["tokens"], W), w, ckv, kpe


def _in_shared(case, seed):
    d = Draws(seed)
    return d.bf(case["tokens"], W), d.bf(1024, W, sd=W ** -0.5), d.bf(W, 512, sd=512 ** -0.5), d.bf(1, W, sd=W ** -0.5)


FF = 8192


def _in_ffn(case, seed):
    d, dt = Draws(seed), _dtype(case)
    w = {"gate": d.bf(FF, W, sd=W ** -0.5), "up": d.bf(FF, W, sd=W ** -0.5), "down": d.bf(W, FF, sd=FF ** -0.5)}
    return d.n(case["tokens"], W).to(dt), w


MOE = (64, 6, 1024, 2048)                    # experts, top, expert ff, shared ff


def _in_moe(case, seed):
    d, (E, _, F, S) = Draws(seed), MOE
    w = {"router": d.bf(E, W, sd=W ** -0.5), "shared_gate": d.bf(S, W, sd=W ** -0.5), "shared_up": d.bf(S, W, sd=W ** -0.5),
         "shared_down": d.bf(W, S, sd=S ** -0.5)}
    for e in range(E):
        w.update({f"e{e}_gate": d.bf(F, W, sd=W ** -0.5), f"e{e}_up": d.bf(F, W, sd=W ** -0.5), f"e{e}_down": d.bf(W, F, sd=F ** -0.5)})
    return d.n(case["tokens"], W).to(_dtype(case)), w


def _delta_weights(d):
    H, G, n = 32, 16, 128
    w = {"g": d.bf(H * n, W, sd=W ** -0.5), "a": d.bf(H, W, sd=W ** -0.5), "b": d.bf(H, W, sd=W ** -0.5),
         "A_log": torch.log(d.uniform(1.0, 8.0, H)).to(BF), "dt_bias": d.bf(H, mean=-3.0), "norm": d.bf(n, sd=0.1, mean=1.0),
         "o": d.bf(W, H * n, sd=(H * n) ** -0.5)}
    for nm, rows in (("q", G * n), ("k", G * n), ("v", H * n)):
        w[nm], w[nm + "_conv"] = d.bf(rows, W, sd=W ** -0.5), d.bf(rows, 4, sd=0.5)
    return w


def _in_delta(case, seed):
    d = Draws(seed)
    return d.n(case["tokens"], W).to(_dtype(case)), _delta_weights(d)


ATT = (16, 2, 128)                           # heads, kv heads, head size
PAGE = 64


def _requests(case):
    """(new tokens, cached tokens) of every request of a mixed step."""
    return [(case["tokens"], case["past"])] + [(1, case["context"] + 17 * i) for i in range(case["decoding"])]


def _in_attention(case, seed):
    d, dt, (H, G, n) = Draws(seed), _dtype(case), ATT
    w = {"q": d.bf(H * n, W, sd=W ** -0.5), "k": d.bf(G * n, W, sd=W ** -0.5), "v": d.bf(G * n, W, sd=W ** -0.5),
         "q_norm": d.bf(n, sd=0.1, mean=1.0), "k_norm": d.bf(n, sd=0.1, mean=1.0), "o": d.bf(W, H * n, sd=(H * n) ** -0.5)}
    reqs = _requests(case)
    pages, at = [], 0
    for new, past in reqs:
        k = (new + past + PAGE - 1) // PAGE
        pages.append(list(range(at, at + k)))
        at += k
    kc, vc = (d.n(at, PAGE, G * n).to(dt) for _ in range(2))
    return d.n(sum(r[0] for r in reqs), W).to(dt), w, kc, vc, reqs, pages


# the serving benchmark's delta / latent-attention stack without its looped span
SERVE_DELTA = {"heads": 32, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4}
SERVE_LATENT = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "mask": {"size": 1024},
                "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
SERVE_VOCAB = 32768


def _serve_raw():
    dense = {"kind": "dense", "ff": FF}
    layers = [{"type": "delta", "mixer": SERVE_DELTA, "mlp": None}, {"type": "delta", "mixer": SERVE_DELTA, "mlp": dense},
              {"type": "latent_attention", "mixer": SERVE_LATENT, "mlp": dense}]
    return {"architecture": "Vofelix", "vocab": SERVE_VOCAB, "width": W, "embedding": {"scale": 8.0}, "norm": {"eps": 1e-5},
            "token_side": {"dim": 256}, "layers": layers}


def _in_serve(case, seed):
    d = Draws(seed)
    raw, side = _serve_raw(), 256
    w = {"embed": d.bf(SERVE_VOCAB, W, sd=0.125), "head": d.bf(SERVE_VOCAB, W, sd=W ** -0.5), "final.norm": d.bf(W, sd=0.1, mean=1.0),
         "final.norm.b": d.bf(W, sd=0.05), "side.embed": d.bf(SERVE_VOCAB, 3 * side)}
    for i, L in enumerate(raw["layers"]):
        p = f"l{i}."
        for nm in ("norm1", "norm1b") + (("norm2", "norm2b") if L["mlp"] else ()):
            w[p + nm], w[p + nm + ".b"] = d.bf(W, sd=0.1, mean=1.0), d.bf(W, sd=0.05)
        if L["type"] == "delta":
            w.update({p + "mix." + k.replace("_conv", ".conv"): v for k, v in _delta_weights(d).items()})
        else:
            w.update({p + "mix.q": d.bf(16 * 192, W, sd=W ** -0.5), p + "mix.dkv": d.bf(576, W, sd=W ** -0.5), p + "mix.dkv.norm": d.bf(512, sd=0.1, mean=1.0),
                      p + "mix.uk": d.bf(2048, 512, sd=512 ** -0.5), p + "mix.uv": d.bf(2048, 512, sd=512 ** -0.5), p + "mix.sink": d.bf(16),
                      p + "mix.o": d.bf(W, 2048, sd=W ** -0.5)})
        if L["mlp"]:
            w.update({p + "mlp.gate": d.bf(FF, W, sd=W ** -0.5), p + "mlp.up": d.bf(FF, W, sd=W ** -0.5), p + "mlp.down": d.bf(W, FF, sd=FF ** -0.5)})
        w.update({p + "side.gate": d.bf(side, W, sd=W ** -0.5), p + "side.proj": d.bf(W, side, sd=side ** -0.5), p + "side.norm": d.bf(W, sd=0.1, mean=1.0)})
    prompts = [d.ints(0, SERVE_VOCAB, case["prompt"] + 3 * i).tolist() for i in range(case["requests"])]
    fed = d.ints(0, SERVE_VOCAB, case["decode"], case["requests"]).tolist()
    return raw, w, prompts, fed


# ------------------------------------------------------------------------------------------------ prepare / run

def prepare(case, seed):
    kind, s = case["kind"], types.SimpleNamespace(case=case)
    if kind == "experts":
        from krasis_b200 import GpuPrefillManager, KrasisEngine
        E, k, I, renorm = EXPERTS[case["model"]]
        t = _in_experts(case, seed)
        s.x = t["x"]
        s.engine = KrasisEngine(hidden_size=W, moe_intermediate_size=I, n_routed_experts=E, num_experts_per_tok=k, num_moe_layers=1,
                                num_bits=case["bits"], norm_topk_prob=renorm, max_tokens=MAXT)
        s.engine.load_quantized_layer_dev(0, t["w13_q"], t["w13_s"].view(torch.int16), t["w2_q"], t["w2_s"].view(torch.int16))
        s.engine.set_routing_weights(0, t["gate"])
        s.manager = GpuPrefillManager(krasis_engine=s.engine, num_bits=case["bits"], max_tokens=MAXT)
    elif kind == "deltanet":
        from krasis_b200.attention import GatedDeltaNetAttention
        s.x, w = _in_deltanet(case, seed)
        s.layer = GatedDeltaNetAttention(DN, 0, w, DEV, max_tokens=MAXT)
    elif kind in ("gqa", "mla"):
        from krasis_b200 import attention as A
        total = case["past"] + case["tokens"]
        pages = (total + 15) // 16
        if kind == "gqa":
            s.x, w, k, v = _in_gqa(case, seed)
            s.layer, s.cache = A.GQAAttention(GQA, 0, w, DEV, max_tokens=MAXT), A.PagedKVCache(1, 2, 256, DEV, pages + 1)
            pools = (s.cache.k_cache[0].view(-1, 512), s.cache.v_cache[0].view(-1, 512))
        else:
            s.x, w, k, v = _in_mla(case, seed)
            s.layer, s.cache = A.MLAAttention(MLA, 0, w, DEV, max_tokens=MAXT, max_kv_len=MAXT), A.MLAPagedKVCache(1, 512, 64, DEV, pages + 1)
            pools = (s.cache.ckv_cache[0].view(-1, 512), s.cache.kpe_cache[0].view(-1, 64))
        s.seq = A.SequenceKVState(s.cache)
        s.seq.ensure_capacity(total)
        rows = torch.tensor(s.seq.pages, device=DEV).repeat_interleave(16)[:total] * 16 + torch.arange(total, device=DEV) % 16
        past = case["past"]
        for pool, t in zip(pools, (k, v)):                                    # the keys of the earlier portions
            pool.view(torch.uint8)[rows[:past]] = t.view(torch.uint8)[:past]
        s.seq.advance(past)
        s.positions = torch.arange(past, total, dtype=torch.int32, device=DEV)
    elif kind == "shared":
        from krasis_b200.layers import SharedExpert
        s.x, gu, down, gate = _in_shared(case, seed)
        s.layer = SharedExpert(gu, down, gate)
    elif kind == "ffn":
        from krasis_b200.mixers import GatedMLP
        s.x, w = _in_ffn(case, seed)
        s.layer = GatedMLP(w, _dtype(case), DEV, act=case["act"])
    elif kind == "moe":
        from krasis_b200.mixers import RoutedExperts
        s.x, w = _in_moe(case, seed)
        s.layer = RoutedExperts(w, MOE[0], 0, MOE[1], _dtype(case), DEV, score="softmax", renorm=True, act="silu")
    elif kind == "delta":
        from krasis_b200 import seqops
        from krasis_b200.attention import RecurrentStatePool
        from krasis_b200.mixers import GatedDeltaMixer
        s.x, w = _in_delta(case, seed)
        s.layer = GatedDeltaMixer(w, 32, 16, 128, 128, 4, 1e-5, _dtype(case), DEV)
        s.tail, s.state = s.layer.register_state(RecurrentStatePool(4, DEV))
        s.tables = seqops.StepTables([([0] * case["tokens"], 0, 1, [0])], DEV)
    elif kind == "attention":
        from krasis_b200 import seqops
        from krasis_b200.mixers import MultiMapAttention
        s.x, w, s.kc, s.vc, reqs, pages = _in_attention(case, seed)
        H, G, n = ATT
        s.layer = MultiMapAttention(w, H, G, 1, n, n, n ** -0.5, 1e-5, _dtype(case), DEV, window=case["window"] or None, rot_dims=64, rot_base=10000.0)
        s.tables = seqops.StepTables([([0] * new, past, i, pg) for i, ((new, past), pg) in enumerate(zip(reqs, pages))], DEV)
    else:
        from krasis_b200.scheduler import Scheduler
        from krasis_b200.vofelix import VofelixConfig, VofelixModel
        raw, w, s.prompts, s.fed = _in_serve(case, seed)
        model = VofelixModel(VofelixConfig.from_dict(raw), w, dtype=_dtype(case))
        most = case["prompt"] + 3 * case["requests"] + case["decode"]
        s.scheduler = Scheduler(model, max_tokens=case["requests"] * ((most + PAGE - 1) // PAGE) * PAGE, max_requests=case["requests"], cuda_graphs=True)
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "experts":
        ids, wts = s.engine.compute_routing(0, s.x)
        return {"ids": ids, "weights": wts, "out": s.manager.forward(0, s.x, ids, wts)}
    if kind == "deltanet":
        s.layer.reset_state()                                                  # a new prompt
        return {"out": s.layer.forward(s.x)}
    if kind in ("gqa", "mla"):
        return {"out": s.layer.forward(s.x, s.positions, s.cache, s.seq, 0, case["tokens"])}
    if kind in ("shared", "ffn", "moe"):
        return {"out": s.layer.forward(s.x)}
    if kind == "delta":
        s.tail[1].zero_()                                                      # what handing out a state slot does
        s.state[1].zero_()
        return {"out": s.layer.forward(s.x, s.tables, s.tail, s.state), "tail": s.tail[1], "state": s.state[1]}
    if kind == "attention":
        return {"out": s.layer.forward(s.x, s.tables, s.kc, s.vc, PAGE)}
    sched, n = s.scheduler, case["requests"]
    # prompts arrive together, cut so that a step carries at most 256 of their tokens; then every request decodes given tokens
    first = []
    at = [0] * n
    while any(at[i] < len(p) for i, p in enumerate(s.prompts)):
        budget, entries, done = 256, [], []
        for i, p in enumerate(s.prompts):
            k = min(budget, len(p) - at[i])
            if k > 0:
                at[i] += k
                budget -= k
                entries.append((i, p[at[i] - k:at[i]], [k - 1] if at[i] == len(p) else []))
        logits = sched.step(entries)
        if logits is not None:
            first.append(logits)
    for row in s.fed:
        logits = sched.step([(i, [row[i]], [0]) for i in range(n)])
    for i in range(n):
        sched.finish(i)
    return {"first": torch.cat(first, 0), "last": logits}


# ------------------------------------------------------------------------------------------------ work

def work(case):
    """Inputs, weights that the pass touches, caches and outputs once each; multiply-adds of the products as two operations."""
    kind, T = case["kind"], case.get("tokens", 0)
    if kind == "experts":
        E, k, I, _ = EXPERTS[case["model"]]
        touched = E * (1.0 - (1.0 - k / E) ** T)
        per = 3 * W * I * (case["bits"] / 8 + 2 / 128)
        return {"bytes": touched * per + E * W * 2 + 2 * T * W * 2 + T * k * 8, "flops": 2.0 * T * (k * 3 * W * I + E * W)}
    if kind == "deltanet":
        wts = 12288 * W + 64 * W + 4096 * W
        return {"bytes": 2.0 * (wts + 2 * T * W) + 32 * 128 * 128 * 4, "flops": 2.0 * T * wts + T * 32 * 128 * 128 * 8.0}
    if kind == "gqa":
        wts, pairs = (8192 + 1024) * W + 4096 * W, T * (case["past"] + (T + 1) / 2)
        return {"bytes": 2.0 * (wts + 2 * T * W) + 1024.0 * (case["past"] + T), "flops": 2.0 * T * wts + pairs * 16 * 256 * 4}
    if kind == "mla":
        wts, total = (3072 + 576) * W + 2 * 2048 * 512 + 2048 * W, case["past"] + T
        pairs = T * (case["past"] + (T + 1) / 2)
        return {"bytes": 2.0 * (wts + 2 * T * W) + 576.0 * total, "flops": 2.0 * T * (3648 * W + 2048 * W) + 2.0 * total * 4096 * 512 + pairs * 16 * 320 * 2}
    if kind == "shared":
        wts = 1024 * W + W * 512
        return {"bytes": wts + 4.0 * T * W + 2 * W, "flops": 2.0 * T * wts}
    es = 4 if case["dtype"] == "float32" else 2
    if kind == "ffn":
        return {"bytes": es * 3.0 * W * FF + T * W * (es + 4), "flops": 6.0 * T * W * FF}
    if kind == "moe":
        E, k, F, S = MOE
        touched = E * (1.0 - (1.0 - k / E) ** T)
        return {"bytes": es * (touched * 3 * W * F + 3.0 * W * S + E * W) + T * W * (es + 4), "flops": 2.0 * T * (k * 3 * W * F + 3 * W * S + E * W)}
    if kind == "delta":
        wts = (2 * 2048 + 2 * 4096 + 64) * W + 4096 * W
        return {"bytes": es * float(wts) + T * W * (es + 4) + 32 * 128 * 128 * 4, "flops": 2.0 * T * wts + T * 32 * 128 * 128 * 8.0}
    if kind == "attention":
        H, G, n = ATT
        wts, win = (H * n + 2 * G * n) * W + W * H * n, case["window"] or 1 << 30
        keys = pairs = rows = 0
        for new, past in _requests(case):
            rows += new
            keys += min(past + new, win + new - 1)
            lo, hi = past + 1, past + new                                      # visible keys of the first and last new token
            full = max(0, hi - max(lo, win + 1) + 1)
            part = new - full
            pairs += full * win + part * (lo + lo + part - 1) / 2
        return {"bytes": es * (wts + 2.0 * keys * G * n) + rows * W * (es + 4), "flops": 2.0 * rows * wts + pairs * H * n * 4}
    delta = (2 * 2048 + 2 * 4096 + 64) * W + 4096 * W
    latent = (3072 + 576) * W + 2 * 2048 * 512 + 2048 * W
    layers = 2 * delta + latent + 2 * 3 * W * FF + 3 * 2 * 256 * W
    n = case["requests"]
    prompt = sum(case["prompt"] + 3 * i for i in range(n))
    portions = math.ceil(prompt / 256)
    state = 2 * 2.0 * 32 * 128 * 128 * 4 * 2 * n                               # two delta states per request, read and written once a step
    keys = case["prompt"] + 1.5 * (n - 1) + case["decode"] / 2
    step = 2.0 * (layers + SERVE_VOCAB * W)
    return {"bytes": portions * step + case["decode"] * (step + state + n * keys * 576 * 2.0),
            "flops": 2.0 * (prompt + case["decode"] * n) * layers + 2.0 * n * (case["decode"] + 1) * SERVE_VOCAB * W}


# ------------------------------------------------------------------------------------------------ tolerance

def tolerance(case):
    kind, exactly = case["kind"], case.get("dtype") == "float32"
    if kind == "experts":
        # three bf16 roundings between input and output; a router logit near a tie may pick the neighbour
        return {"rel": 0.012, "max": 0.3, "differ": 0.002}
    if kind in ("gqa", "mla"):
        return {"rel": 0.02, "max": 0.5}                                       # FP8 cache: a bf16 neighbour may move a key by one FP8 step
    if kind == "deltanet":
        return {"rel": 0.02, "max": 0.5}
    if kind == "shared":
        return {"rel": 0.012, "max": 0.3}
    if kind == "serve":
        return {"rel": 0.03, "max": 0.5}                                       # bf16 through three layers of mixers and feed-forwards
    if exactly:
        return {"rel": 1e-5, "max": 4e-4}
    return {"rel": 0.012, "max": 0.3}


# ------------------------------------------------------------------------------------------------ exact (float64)

def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _act(g, act):
    return torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")


def _mm(x, w, step=1024):
    """x @ w^T in float64, w converted a few rows at a time."""
    return torch.cat([x @ w[i:i + step].double().T for i in range(0, w.shape[0], step)], 1)


def _delta_scan(q, k, v, beta, decay):
    """S <- decay S; S += k beta (v - S^T k)^T; o = S^T q.  q, k [T, H, dk], v [T, H, dv], beta, decay [T, H]."""
    T, H, dk = q.shape
    S, out = torch.zeros(H, dk, v.shape[2], dtype=torch.float64, device=q.device), torch.empty_like(v)
    for t in range(T):
        S *= decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S.baddbmm_(k[t][:, :, None], u[:, None])
        out[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return out, S


def _conv_silu(x, taps):
    """Causal convolution per channel over time, then SiLU.  x [T, C], taps [C, K]."""
    K, pad = taps.shape[1], torch.zeros(taps.shape[1] - 1, x.shape[1], dtype=x.dtype, device=x.device)
    xp = torch.cat([pad, x], 0)
    return torch.nn.functional.silu(sum(xp[i:i + x.shape[0]] * taps[:, i].double() for i in range(K)))


def _unit(x, eps):
    return x * torch.rsqrt(x.square().sum(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, start, window=1 << 30):
    """Causal attention of rows q [T, H, d] at positions start.. over k [L, G, d], v [L, G, dv]."""
    T, H, _ = q.shape
    G, L = k.shape[1], k.shape[0]
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device=q.device)
    key = torch.arange(L, device=q.device)
    for t0 in range(0, T, 256):
        pos = start + torch.arange(t0, min(T, t0 + 256), device=q.device)
        away = pos[:, None] - key[None]
        hide = (away < 0) | (away >= window)
        for h in range(H):
            g = h * G // H
            s = (q[t0:t0 + 256, h] @ k[:, g].T * scale).masked_fill(hide, float("-inf"))
            out[t0:t0 + 256, h] = torch.softmax(s, -1) @ v[:, g]
    return out


def _exact_experts(case, seed):
    t = _in_experts(case, seed)
    E, k, I, renorm = EXPERTS[case["model"]]
    x = t["x"].double()
    p = torch.softmax(x @ t["gate"].double().T, -1)
    wts, ids = torch.topk(p, k, -1)
    if renorm:
        wts = wts / wts.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(E):
        tok, j = torch.nonzero(ids == e, as_tuple=True)
        if not tok.numel():
            continue
        gu = x[tok] @ _dequant(t["w13_q"][e], t["w13_s"][e], case["bits"]).T
        y = (torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]) @ _dequant(t["w2_q"][e], t["w2_s"][e], case["bits"]).T
        out.index_add_(0, tok, y * wts[tok, j][:, None])
    return {"ids": ids.to(torch.int32), "weights": wts, "out": out}


def _exact_deltanet(case, seed):
    x, w = _in_deltanet(case, seed)
    T, x = x.shape[0], x.double()
    qkvz = _mm(x, w["in_proj_qkvz"]).view(T, 16, 768)
    ba = _mm(x, w["in_proj_ba"]).view(T, 16, 4)
    q, k, v, z = qkvz[..., :128], qkvz[..., 128:256], qkvz[..., 256:512], qkvz[..., 512:].reshape(T, 32, 128)
    b, a = ba[..., :2].reshape(T, 32), ba[..., 2:].reshape(T, 32)
    c = _conv_silu(torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], 1), w["conv1d_weight"][:, 0])
    q, k, v = c[:, :2048].view(T, 16, 128), c[:, 2048:4096].view(T, 16, 128), c[:, 4096:].view(T, 32, 128)
    q, k = _unit(q, 1e-6).repeat_interleave(2, 1) * 128 ** -0.5, _unit(k, 1e-6).repeat_interleave(2, 1)
    decay = torch.exp(-torch.exp(w["A_log"].double()) * torch.nn.functional.softplus(a + w["dt_bias"].double()))
    o, _ = _delta_scan(q, k, v, torch.sigmoid(b), decay)
    o = _rms(o, w["norm_weight"], 1e-6) * torch.nn.functional.silu(z)
    return {"out": _mm(o.reshape(T, -1), w["out_proj"])}


def _half_rope(x, pos, freq):
    """Dimension i turns with i + d / 2 (bf16 angle tables, as the models define them)."""
    ang = (pos.float()[:, None] * freq.float()[None]).to(torch.float32)
    c, s = ang.cos().to(BF).double()[:, None], ang.sin().to(BF).double()[:, None]
    h = freq.numel()
    a, b = x[..., :h], x[..., h:2 * h]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * h:]], -1)


def _fp8(x):
    """The value a cache byte holds: bf16 rows cast to FP8."""
    return x.to(BF).to(torch.float8_e4m3fn).double()


def _exact_gqa(case, seed):
    x, w, kc, vc = _in_gqa(case, seed)
    T, past, x = case["tokens"], case["past"], x.double()
    pos = torch.arange(past, past + T, device=DEV)
    freq = 1.0 / (GQA.rope_theta ** (torch.arange(0, 64, 2, device=DEV).float() / 64))
    q = _mm(x, w["q_proj"]).view(T, 16, 512)
    gate, q = q[..., 256:], _half_rope(_rms(q[..., :256], w["q_norm"], 1e-6), pos, freq)
    k = _half_rope(_rms(_mm(x, w["k_proj"]).view(T, 2, 256), w["k_norm"], 1e-6), pos, freq)
    v = _mm(x, w["v_proj"]).view(T, 2, 256)
    k = torch.cat([kc[:past].double().view(-1, 2, 256), _fp8(k)])
    v = torch.cat([vc[:past].double().view(-1, 2, 256), _fp8(v)])
    o = _attend(q, k, v, 1 / 16, past) * torch.sigmoid(gate)
    return {"out": _mm(o.reshape(T, -1), w["o_proj"])}


def _exact_mla(case, seed):
    x, w, cc, pc = _in_mla(case, seed)
    T, past, x = case["tokens"], case["past"], x.double()
    pos = torch.arange(past, past + T, device=DEV)
    dim, base, orig, factor = 64, MLA.rope_theta, 4096, 40.0
    freq = 1.0 / (base ** (torch.arange(0, dim, 2, device=DEV).float() / dim))
    turn = lambda beta: dim * math.log(orig / (beta * 2 * math.pi)) / (2 * math.log(base))  # noqa: E731
    low, high = max(math.floor(turn(32)), 0), min(math.ceil(turn(1)), dim // 2 - 1)
    mask = 1.0 - torch.clamp((torch.arange(dim // 2, device=DEV).float() - low) / max(high - low, 0.001), 0, 1)
    freq = freq / factor * (1 - mask) + freq * mask
    scale = 192 ** -0.5 * (0.1 * 0.707 * math.log(factor) + 1.0) ** 2

    def rope(t):                                                               # interleaved pairs side by side, then the half-split turn
        return _half_rope(t.unflatten(-1, (32, 2)).transpose(-1, -2).reshape(t.shape), pos, freq)
    q = _mm(x, w["q_proj"]).view(T, 16, 192)
    kv = _mm(x, w["kv_a_proj_with_mqa"])
    ckv = torch.cat([cc[:past].double(), _fp8(_rms(kv[:, :512], w["kv_a_layernorm"], 1e-6))])
    kpe = torch.cat([pc[:past].double(), _fp8(rope(kv[:, None, 512:])[:, 0])])
    k = torch.cat([torch.einsum("lr,hnr->lhn", ckv, w["w_kc"].double()), kpe[:, None].expand(-1, 16, -1)], -1)
    v = torch.einsum("lr,hvr->lhv", ckv, w["w_vc"].double())
    o = _attend(torch.cat([q[..., :128], rope(q[..., 128:])], -1), k, v, scale, past)
    return {"out": _mm(o.reshape(T, -1), w["o_proj"])}


def _int8_rows(x):
    s = (x.float().abs().amax(-1, keepdim=True) / 127.0).clamp_min(1e-10)
    return torch.round(x.float() / s).clamp(-127, 127).double(), s


def _exact_shared(case, seed):
    x, gu, down, gate = _in_shared(case, seed)

    def lin8(a, w):
        (aq, sa), (wq, sw) = _int8_rows(a), _int8_rows(w)
        return (aq @ wq.T) * sa.double() * sw.to(BF).double().T
    h = lin8(x, gu).to(BF).double()
    a = (torch.nn.functional.silu(h[:, :512]) * h[:, 512:]).to(BF)              # quantised per row ahead of the second product
    return {"out": lin8(a, down) * torch.sigmoid(x.double() @ gate.double().T)}


def _exact_ffn(case, seed):
    x, w = _in_ffn(case, seed)
    x = x.double()
    return {"out": _mm(_act(_mm(x, w["gate"]), case["act"]) * _mm(x, w["up"]), w["down"])}


def _exact_moe(case, seed):
    x, w = _in_moe(case, seed)
    x = x.double()
    p, ids = torch.topk(torch.softmax(_mm(x, w["router"]), -1), MOE[1], -1)
    p = p / p.sum(-1, keepdim=True)
    silu = torch.nn.functional.silu
    out = _mm(silu(_mm(x, w["shared_gate"])) * _mm(x, w["shared_up"]), w["shared_down"])
    for e in range(MOE[0]):
        tok, j = torch.nonzero(ids == e, as_tuple=True)
        if tok.numel():
            y = _mm(silu(_mm(x[tok], w[f"e{e}_gate"])) * _mm(x[tok], w[f"e{e}_up"]), w[f"e{e}_down"])
            out.index_add_(0, tok, y * p[tok, j][:, None])
    return {"out": out}


def _exact_delta(case, seed):
    x, w = _in_delta(case, seed)
    T, x, H = x.shape[0], x.double(), 32
    raw = torch.cat([_mm(x, w[n]) for n in ("q", "k", "v")], 1)
    c = _conv_silu(raw, torch.cat([w[n + "_conv"] for n in ("q", "k", "v")], 0))
    q, k, v = c[:, :2048].view(T, 16, 128), c[:, 2048:4096].view(T, 16, 128), c[:, 4096:].view(T, H, 128)
    q, k = _unit(q, 1e-6).repeat_interleave(2, 1) * 128 ** -0.5, _unit(k, 1e-6).repeat_interleave(2, 1)
    decay = torch.exp(-torch.exp(w["A_log"].double()) * torch.nn.functional.softplus(_mm(x, w["a"]) + w["dt_bias"].double()))
    o, S = _delta_scan(q, k, v, torch.sigmoid(_mm(x, w["b"])), decay)
    o = _rms(o, w["norm"], 1e-5) * torch.nn.functional.silu(_mm(x, w["g"])).view(T, H, 128)
    tail = torch.cat([torch.zeros(3, raw.shape[1], dtype=raw.dtype, device=DEV), raw])[-3:].T
    return {"out": _mm(o.reshape(T, -1), w["o"]), "tail": tail, "state": S}


def _exact_attention(case, seed):
    x, w, kc, vc, reqs, pages = _in_attention(case, seed)
    H, G, n = ATT
    freq = 10000.0 ** (-torch.arange(0, 64, 2, device=DEV, dtype=torch.float64) / 64)

    def turn(t, pos):                                                          # dimension 2i with 2i + 1
        ang = pos.double()[:, None, None] * freq
        a, b = t[..., 0:64:2], t[..., 1:64:2]
        r = torch.stack([a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()], -1).flatten(-2)
        return torch.cat([r, t[..., 64:]], -1)
    o, at, x, stored = [], 0, x.double(), kc.dtype
    for (new, past), pg in zip(reqs, pages):
        h, pos = x[at:at + new], torch.arange(past, past + new, device=DEV)
        at += new
        q = turn(_rms(_mm(h, w["q"]).view(new, H, n), w["q_norm"], 1e-5), pos)
        k = turn(_rms(_mm(h, w["k"]).view(new, G, n), w["k_norm"], 1e-5), pos)
        v = _mm(h, w["v"]).view(new, G, n)
        old = [t[pg].reshape(-1, G, n)[:past].double() for t in (kc, vc)]
        k, v = (torch.cat([a, b.to(stored).double()]) for a, b in zip(old, (k, v)))
        o.append(_attend(q, k, v, n ** -0.5, past, case["window"] or 1 << 30))
    return {"out": _mm(torch.cat(o).reshape(at, -1), w["o"])}


def exact(case, seed):
    if case["kind"] == "serve":
        return None                                                            # a whole model over many steps: its layers are cases of their own
    return globals()["_exact_" + case["kind"]](case, seed)
