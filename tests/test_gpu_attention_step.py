"""An attention layer's step in one C call launches what the calls one by one launch: the same bits, in outputs and caches."""
import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = [[(200, 0), (1, 700)], [(1, 90), (150, 10), (1, 300), (3, 2000)], [(128, 0), (130, 5)], [(1, 0)], [(127, 1), (2, 63)]]


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("dtype,dv,window,extra", [
    (torch.bfloat16, 128, 512, {}), (torch.bfloat16, 256, None, {"softcap": 30.0}), (torch.bfloat16, 128, 100, {"slopes": True, "bias": True}),
    (torch.bfloat16, 64, 512, {"sink": True}), (torch.float32, 128, 130, {"norm": True, "sink": True}), (torch.bfloat16, 128, None, {"kv_one": True, "norm": True}),
])
def test_step_matches_single_calls(step, dtype, dv, window, extra, monkeypatch):
    from krasis_b200 import seqops as ops
    from krasis_b200.mixers import MultiMapAttention
    W, H, G, d = 256, 6, 2, 128
    g = torch.Generator().manual_seed(9)
    r = lambda *s, sd=W ** -0.5: torch.randn(*s, generator=g) * sd  # noqa: E731
    w, kw = {"q": r(H * d, W), "k": r(G * d, W), "v": r(G * dv, W), "o": r(W, H * dv, sd=(H * dv) ** -0.5)}, {}
    if extra.get("kv_one"):
        del w["v"]
        kw["keys_as_values"] = True
    if extra.get("bias"):
        w["q_b"] = r(H * d, sd=1.0)
    if extra.get("sink"):
        w["sink"] = r(H, sd=1.0)
    if extra.get("norm"):
        w["q_norm"], w["k_norm"] = 1 + r(d, sd=0.1), 1 + r(d, sd=0.1)
    if extra.get("slopes"):
        kw["slopes"] = 2.0 ** -torch.arange(1, H + 1)
    m = MultiMapAttention(w, H, G, 1, d, dv, d ** -0.5, 1e-5, dtype, "cuda", window=window, rot_dims=64, softcap=extra.get("softcap", 0.0), **kw)
    entries, page = [], 0
    for i, (n, past) in enumerate(step):
        k = (n + past + 63) // 64
        entries.append(([0] * n, past, i, list(range(page, page + k))[::-1]))
        page += k
    tb = ops.StepTables(entries, "cuda")
    kc, vc = (torch.randn(page, 64, c, generator=g).to(dtype).cuda() for c in (G * d, G * dv))
    h = torch.randn(tb.T, W, generator=g).to(dtype).cuda()
    assert m._one_call()
    k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    got = m.forward(h, tb, k1, v1, 64)
    monkeypatch.setattr(MultiMapAttention, "_one_call", lambda self: False)
    want = m.forward(h, tb, k2, v2, 64)
    assert torch.equal(got, want) and torch.equal(k1, k2) and torch.equal(v1, v2)
    assert bool(torch.isfinite(got).all())


def test_pages_that_do_not_hold_a_portion():
    from krasis_b200 import seqops as ops
    from krasis_b200.mixers import MultiMapAttention
    g = torch.Generator().manual_seed(9)
    r = lambda *s: torch.randn(*s, generator=g) * 0.05  # noqa: E731
    m = MultiMapAttention({"q": r(256, 256), "k": r(128, 256), "v": r(128, 256), "o": r(256, 256)}, 2, 1, 1, 128, 128, 0.1, 1e-5, torch.bfloat16, "cuda")
    tb = ops.StepTables([([0] * 130, 0, 0, [0, 1, 2])], "cuda")
    tb.layout = [(0, 130, 64, [0, 1, 2])]                    # says 194 positions: 4 pages; nothing may be launched
    kc = torch.zeros(4, 64, 128, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(IndexError):
        m.forward(torch.zeros(130, 256, dtype=torch.bfloat16, device="cuda"), tb, kc, kc.clone(), 64)
    assert not kc.any()


@pytest.mark.parametrize("least", [0, 1, 5])
def test_shortest_portion_of_the_tensor_cores(least, monkeypatch):
    """tc_min_portion: 0 and 1 send every portion to the tensor cores, in one call as in single ones."""
    from krasis_b200 import seqops as ops
    from krasis_b200.mixers import MultiMapAttention
    g = torch.Generator().manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g) * 0.06  # noqa: E731
    m = MultiMapAttention({"q": r(512, 256), "k": r(128, 256), "v": r(128, 256), "o": r(256, 512)}, 4, 1, 1, 128, 128, 128 ** -0.5, 1e-5, torch.bfloat16, "cuda")
    m.tc_min_portion = least
    tb = ops.StepTables([([0] * 3, 20, 0, [0]), ([0], 70, 1, [2, 1]), ([0] * 140, 0, 2, [3, 4, 5])], "cuda")
    kc, vc = (torch.randn(6, 64, 128, generator=g).bfloat16().cuda() for _ in range(2))
    h = torch.randn(tb.T, 256, generator=g).bfloat16().cuda()
    portions = []
    portion_rows = ops.portion_rows
    monkeypatch.setattr(ops, "portion_rows", lambda tb, s, *a: portions.append(s) or portion_rows(tb, s, *a))
    got = m.forward(h, tb, kc.clone(), vc.clone(), 64)
    assert not portions and m._one_call()
    monkeypatch.setattr(MultiMapAttention, "_one_call", lambda self: False)
    want = m.forward(h, tb, kc, vc, 64)
    assert torch.equal(got, want) and portions == {0: [0, 1, 2], 1: [0, 1, 2], 5: [2]}[least]
