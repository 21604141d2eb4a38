"""The delta rule sixteen tokens at a time, the short convolution's vector form and the gated read-out at their edges, against fp64."""
import pytest
import torch

from krasis_b200 import seqops as ops

pytestmark = pytest.mark.gpu


def _mixer(H, Hk, dk, dv, dtype=torch.float32, decay=-3.0):
    from krasis_b200.mixers import GatedDeltaMixer
    W = 64
    g = torch.Generator().manual_seed(H + dk + dv)
    r = lambda *s, sd=W ** -0.5: torch.randn(*s, generator=g) * sd  # noqa: E731
    w = {"q": r(Hk * dk, W), "k": r(Hk * dk, W), "v": r(H * dv, W), "g": r(H * dv, W), "a": r(H, W), "b": r(H, W), "A_log": r(H, sd=0.5),
         "dt_bias": r(H, sd=1.0) + decay, "norm": 1 + r(dv, sd=0.1), "o": r(W, H * dv, sd=(H * dv) ** -0.5)}
    for n, c in (("q", Hk * dk), ("k", Hk * dk), ("v", H * dv)):
        w[n + "_conv"] = r(c, 4, sd=0.5)
    return GatedDeltaMixer(w, H, Hk, dk, dv, 4, 1e-5, dtype, "cuda")


def _exact(m, h, tb, tail, state, lens, slots):
    """State and output in fp64, token by token."""
    H, Hk, dk, dv = m.H, m.Hk, m.dk, m.dv
    proj = h.double() @ m.w_in.double().T
    outs, states = [], state.double().clone()
    at = 0
    for n, slot in zip(lens, slots):
        raw = torch.cat([tail[slot].double().T, proj[at:at + n, :m.C]], 0)
        c = torch.nn.functional.silu(sum(raw[i:i + n] * m.taps[:, i].double() for i in range(4)))
        q, k, v = c[:, :Hk * dk].view(n, Hk, dk), c[:, Hk * dk:2 * Hk * dk].view(n, Hk, dk), c[:, 2 * Hk * dk:].view(n, H, dv)
        unit = lambda x: x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k = unit(q).repeat_interleave(H // Hk, 1) * dk ** -0.5, unit(k).repeat_interleave(H // Hk, 1)
        p = proj[at:at + n]
        dec = torch.exp(-torch.exp(m.A_log.double()) * torch.nn.functional.softplus(p[:, m.a_off:m.a_off + H] + m.dt_bias.double()))
        beta = torch.sigmoid(p[:, m.b_off:m.b_off + H])
        S = states[slot]
        o = torch.empty(n, H, dv, dtype=torch.float64, device=h.device)
        for t in range(n):
            S = S * dec[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None]
            o[t] = torch.einsum("hkv,hk->hv", S, q[t])
        states[slot] = S
        o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + 1e-5) * m.norm.double()
        outs.append((o * torch.nn.functional.silu(p[:, m.g_off:m.g_off + H * dv].reshape(n, H, dv))).reshape(n, -1) @ m.w_o.double().T)
        at += n
    return torch.cat(outs), states


# portions that end anywhere in a tile of sixteen, one-token portions beside long ones, an odd number of slices and heads per key head
@pytest.mark.parametrize("H,Hk,dk,dv", [(2, 1, 32, 32), (4, 4, 64, 96), (6, 2, 128, 64), (9, 1, 32, 32)])
@pytest.mark.parametrize("lens", [[16], [17, 1, 18], [1, 31, 2, 3], [64, 67], [71, 70, 69, 68], [15, 33], [79, 80, 81], [96, 1, 95]])
@pytest.mark.parametrize("decay", [-3.0, 3.0])                 # slow, and so fast that a tile forgets all it knew
def test_tiles_against_exact_and_token_form(H, Hk, dk, dv, lens, decay):
    m = _mixer(H, Hk, dk, dv, decay=decay)
    g = torch.Generator(device="cuda").manual_seed(7)
    slots = [(3 * i + 2) % 5 for i in range(len(lens))]
    tb = ops.StepTables([([0] * n, 0 if i else 9, s, [0]) for i, (n, s) in enumerate(zip(lens, slots))], "cuda")
    h = torch.randn(sum(lens), 64, device="cuda", generator=g)
    tail0, state0 = torch.randn(5, m.C, 3, device="cuda", generator=g), torch.randn(5, H, dk, dv, device="cuda", generator=g)
    # positions only matter to the convolution's tail: the first rows of a portion read it whatever the position
    want, states = _exact(m, h, tb, tail0, state0, lens, slots)
    err = {}
    for name, least in (("tiles", 1), ("tokens", 1 << 30)):
        m.tile_min_portion = least
        tail, state = tail0.clone(), state0.clone()
        got = m.forward(h, tb, tail, state)
        err[name] = (((got.double() - want).norm() / want.norm()).item(), ((state.double() - states).norm() / states.norm()).item())
        untouched = [i for i in range(5) if i not in slots]
        assert torch.equal(state[untouched], state0[untouched])
    # the same fp32 sums in another order: no further off than the token-by-token form, with room for the luck of a few thousand numbers (measured
    # over these and longer portions: outputs 0.81 to 1.02 times its error, states 0.57 to 1.13 times)
    assert err["tiles"][0] <= 1.05 * err["tokens"][0] and err["tiles"][1] <= 1.2 * err["tokens"][1], err


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens", [[70, 20, 12, 65], [12, 300, 20], [64, 63, 64], [9, 128]])
def test_a_sequence_does_not_depend_on_the_step(lens, dtype):
    """Portions on both sides of the tile form's first length, beside one another and alone: the same numbers bit for bit."""
    m = _mixer(8, 4, 128, 64, dtype)
    g = torch.Generator(device="cuda").manual_seed(9)
    h = torch.randn(sum(lens), 64, device="cuda", generator=g).to(dtype)
    tail0, state0 = torch.randn(5, m.C, 3, device="cuda", generator=g), torch.randn(5, 8, 128, 64, device="cuda", generator=g)

    def run(rows, entries):
        tail, state = tail0.clone(), state0.clone()
        o = m.forward(rows, ops.StepTables(entries, "cuda"), tail, state)
        return o, tail, state
    entries = [([0] * n, 9, s, [0]) for s, n in enumerate(lens)]
    whole, tail, state = run(h, entries)
    want, states = _exact(m, h, ops.StepTables(entries, "cuda"), tail0, state0, lens, list(range(len(lens))))
    # fp32: as above; bfloat16: one rounding (2^-9 at most, 2^-9 / sqrt 3 on average) of every head's output ahead of the last product
    assert (whole.double() - want).norm() <= (1e-6 if dtype == torch.float32 else 2.0 ** -9) * want.norm()
    assert (state.double() - states).norm() <= 1e-6 * states.norm()
    at = 0
    for s, n in enumerate(lens):
        if dtype == torch.float32 or (n >= 256) == (sum(lens) >= 256):              # bf16 projections take another kernel from 256 rows on
            alone, t1, s1 = run(h[at:at + n].contiguous(), [([0] * n, 9, s, [0])])
            assert torch.equal(state[s], s1[s]) and torch.equal(tail[s], t1[s]) and torch.equal(whole[at:at + n], alone)
        at += n


def _rule(conv, proj, H, Hk, dk, dv, lens, state, tiles=True):
    """The rule alone on given rows of the convolution [T, q | k | v] and the projection [T, gate | decay | write strength]."""
    lib, S, dev = ops.load(), len(lens), conv.device
    T, C = conv.shape
    cu = torch.tensor([sum(lens[:i]) for i in range(S + 1)], dtype=torch.int32, device=dev)
    slots = torch.arange(S, dtype=torch.int32, device=dev)
    g = torch.Generator(device="cuda").manual_seed(11)
    A_log, dt_bias = torch.randn(H, device=dev, generator=g) * 0.5, torch.randn(H, device=dev, generator=g) - 3.0
    norm = torch.ones(dv, device=dev)
    state, out = state.clone(), torch.full((T, H * dv), float("nan"), device=dev)
    n = lib.kb2_seq_delta_tiles_scratch(T, S, H, Hk, dk, dv) if tiles else 2 * T * Hk * dk + 2 * T * H + T * H * dv + 4
    scratch = torch.empty(int(n), device=dev)
    a = (conv.data_ptr(), C, proj.data_ptr(), proj.stride(0), 0, H * dv, H * dv + H, T, S, H, Hk, dk, dv, A_log.data_ptr(), dt_bias.data_ptr(),
         norm.data_ptr(), 1e-5, state.data_ptr(), cu.data_ptr(), slots.data_ptr(), scratch.data_ptr())
    s = torch.cuda.current_stream().cuda_stream
    ops.check(lib.kb2_seq_delta_tiles(*a, int(n), out.data_ptr(), 0, s) if tiles else lib.kb2_seq_delta_rule(*a, out.data_ptr(), 0, s))
    return out.view(T, H, dv), state


@pytest.mark.parametrize("lens", [[3000, 1, 4001, 190], [16, 6500], [1, 1, 6200, 17, 1000]])
def test_tiles_that_go_in_slices(lens):
    """A step whose tiles do not fit the workspace at once, beside sequences that end in one slice or another: each as by itself, bit for bit."""
    H, Hk, dk, dv, T = 32, 16, 128, 128, sum(lens)
    size = lambda n: ops.load().kb2_seq_delta_tiles_scratch(n, 1, H, Hk, dk, dv) - n * H * dv  # noqa: E731
    assert size(T) < 1.1 * size(T // 2)
    g = torch.Generator(device="cuda").manual_seed(T)
    conv, proj = torch.randn(T, 2 * Hk * dk + H * dv, device="cuda", generator=g), torch.randn(T, H * dv + 2 * H, device="cuda", generator=g)
    state = torch.randn(len(lens), H, dk, dv, device="cuda", generator=g)
    got, after = _rule(conv, proj, H, Hk, dk, dv, lens, state)
    at = 0
    for s, n in enumerate(lens):
        here = state[s:s + 1]
        for a in range(0, n, 3200):                              # portions of whole tiles that one slice holds
            m = min(3200, n - a)
            alone, here = _rule(conv[at + a:at + a + m], proj[at + a:at + a + m], H, Hk, dk, dv, [m], here)
            assert torch.equal(got[at + a:at + a + m], alone)
        assert torch.equal(after[s], here[0])
        at += n


@pytest.mark.parametrize("what", ["value", "key", "query", "decay", "strength"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("H,Hk,dk,dv", [(2, 1, 32, 32), (4, 2, 64, 64), (2, 2, 128, 64)])
def test_numbers_of_a_token_reach_no_earlier_one(H, Hk, dk, dv, bad, what):
    """An infinity or a NaN in any place of a tile leaves the tokens before it, the other sequences and (in a value) the other heads alone."""
    lens, first = [19, 13], 19
    g = torch.Generator(device="cuda").manual_seed(H + dk)
    T = sum(lens)
    conv, proj = torch.randn(T, 2 * Hk * dk + H * dv, device="cuda", generator=g), torch.randn(T, H * dv + 2 * H, device="cuda", generator=g)
    state = torch.randn(2, H, dk, dv, device="cuda", generator=g)
    want, _ = _rule(conv, proj, H, Hk, dk, dv, lens, state)
    assert torch.isfinite(want).all()
    for t in (0, 3, 6, 7, 8, 15, 17, 18):
        c, p = conv.clone(), proj.clone()
        if what in ("decay", "strength"):
            p[t, H * dv + (H if what == "strength" else 0)] = bad
        else:
            c[t, {"value": 2 * Hk * dk, "key": Hk * dk + 1, "query": 1}[what]] = bad
        got, _ = _rule(c, p, H, Hk, dk, dv, lens, state)
        assert torch.equal(got[:t], want[:t]) and torch.equal(got[first:], want[first:]), t
        if what in ("value", "decay", "strength"):
            assert torch.equal(got[:, 1:], want[:, 1:]), t                        # all of head 0


@pytest.mark.parametrize("big", [3.3895e38, 3.4e38, -3.4e38])
@pytest.mark.parametrize("H,Hk,dk,dv", [(2, 1, 32, 32), (2, 2, 128, 64)])
def test_largest_finite_numbers_stay_finite(H, Hk, dk, dv, big):
    """A state next to the end of fp32 is decayed and updated as the token-by-token form does it."""
    lens = [11]
    g = torch.Generator(device="cuda").manual_seed(dv)
    conv, proj = torch.randn(11, 2 * Hk * dk + H * dv, device="cuda", generator=g), torch.randn(11, H * dv + 2 * H, device="cuda", generator=g)
    proj[:, H * dv + H:] = -40.0                                                  # hardly any writing: the state only decays
    state = torch.randn(1, H, dk, dv, device="cuda", generator=g)
    state[0, :, dk // 2, ::3] = big
    want, want_state = _rule(conv, proj, H, Hk, dk, dv, lens, state, tiles=False)
    got, got_state = _rule(conv, proj, H, Hk, dk, dv, lens, state)
    assert torch.isfinite(want_state).all() and torch.isfinite(got_state).all()
    # decays of 11 tokens multiplied one by one or first together, and writes of e^-40 of the products: 32 roundings at most
    assert ((got_state.double() - want_state.double()).abs() <= 2.0 ** -19 * want_state.double().abs() + 1e-6 * want_state.abs().max().double()).all()
    assert torch.equal(got.isfinite(), want.isfinite())


@pytest.mark.parametrize("K,C", [(2, 64), (3, 36), (4, 1028), (4, 30), (5, 64)])
@pytest.mark.parametrize("lens", [[64], [1, 66, 2, 3, 5, 70], [33, 31, 65]])
@pytest.mark.parametrize("bias,bias_out,act", [(False, False, True), (True, False, False), (True, True, True)])
def test_long_convolution(K, C, lens, bias, bias_out, act):
    g = torch.Generator(device="cuda").manual_seed(C + K)
    T, slots = sum(lens), list(range(len(lens)))[::-1]
    proj, taps = torch.randn(T, C + 8, device="cuda", generator=g), torch.randn(C, K, device="cuda", generator=g)
    b = torch.randn(C, device="cuda", generator=g) if bias else None
    bo = torch.randn(C, device="cuda", generator=g) if bias_out else None
    tail0 = torch.randn(len(lens), C, K - 1, device="cuda", generator=g)
    tb = ops.StepTables([([0] * n, 0, s, [0]) for n, s in zip(lens, slots)], "cuda")
    tail = tail0.clone()
    got = ops.conv(proj, C, taps, b, act, tail, tb, bias_out=bo)
    at = 0
    for n, s in zip(lens, slots):
        x = proj[at:at + n, :C].double() + (b.double() if bias else 0.0)
        x = torch.cat([tail0[s].double().T, x], 0)
        y = sum(x[i:i + n] * taps[:, i].double() for i in range(K)) + (bo.double() if bias_out else 0.0)
        y = torch.nn.functional.silu(y) if act else y
        # K + 1 fp32 additions and an exponential: 2^-20 of the terms
        assert ((got[at:at + n].double() - y).abs() <= 2.0 ** -20 * (sum(x[i:i + n].abs() * taps[:, i].double().abs() for i in range(K)) + 3)).all()
        assert (tail[s].double() - x[-(K - 1):].T).abs().max() <= 2.0 ** -22 * x.abs().max()
        at += n
