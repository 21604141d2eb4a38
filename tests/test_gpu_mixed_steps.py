"""A step that mixes long portions (tensor cores) with short ones (plain kernel, key range cut) in any order gives every sequence what a step of
its own gives it."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (new tokens, cached tokens) per sequence: long and short runs in every position, one-token runs between long ones
STEPS = [[(200, 0), (1, 700)], [(1, 700), (200, 64)], [(1, 90), (150, 10), (1, 300), (3, 2000)], [(128, 0), (130, 5)], [(5, 0), (1, 1500), (127, 30)]]


def _tables(step):
    from krasis_b200 import seqops as ops
    entries, page = [], 0
    for i, (n, past) in enumerate(step):
        k = (n + past + 63) // 64
        entries.append(([0] * n, past, i, list(range(page, page + k))))
        page += k
    return ops.StepTables(entries, "cuda"), [ops.StepTables([e], "cuda") for e in entries], page


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("extra", [{}, {"sink": True, "pool": 32}, {"slopes": True}, {"gate": True, "maps": 2}])
def test_attention(step, extra):
    from krasis_b200.mixers import MultiMapAttention, portion_runs
    W, H, G, d, maps = 256, 4, 2, 128, extra.get("maps", 1)
    g = torch.Generator().manual_seed(5)
    r = lambda *s, sd=W ** -0.5: (torch.randn(*s, generator=g) * sd).bfloat16()  # noqa: E731
    w = {"q": r(H * maps * d, W), "k": r(G * maps * d, W), "v": r(G * d, W), "o": r(W, H * d, sd=(H * d) ** -0.5)}
    kw = {}
    if extra.get("sink"):
        w["sink"], kw["pool"] = r(H, sd=1.0), extra["pool"]
    if extra.get("slopes"):
        kw["slopes"] = 2.0 ** -torch.arange(1, H + 1)
    if extra.get("gate"):
        w["g"], kw["map_coef"] = r(H, W), [1.0, -0.4]
    m = MultiMapAttention(w, H, G, maps, d, d, d ** -0.5, 1e-5, torch.bfloat16, "cuda", window=512, rot_dims=64, **kw)
    tb, alone, pages = _tables(step)
    kc, vc = (torch.randn(pages, 64, c, generator=g).bfloat16().cuda() for c in (G * maps * d, G * d))
    pooled = tuple(torch.randn(pages, 2, c, generator=g).bfloat16().cuda() for c in (G * d, G * d)) if "pool" in kw else None
    h = torch.randn(tb.T, W, generator=g).bfloat16().cuda()
    runs = portion_runs(tb, 128)
    assert sum(x[3] for x in runs) == tb.T and [i for x in runs for i in x[1]] == list(range(tb.S))
    got = m.forward(h, tb, kc, vc, 64, pooled=pooled)
    for (row0, n, _, _), one in zip(tb.layout, alone):
        want = m.forward(h[row0:row0 + n].contiguous(), one, kc, vc, 64, pooled=pooled)
        # another cut of the keys and another product kernel for the projections: fp32 rounding (1e-6) ahead of the bf16 rounding of the
        # heads, which then may fall to the other side in places: half a bf16 step of the norm bounds it
        assert (got[row0:row0 + n] - want).norm() <= 2.0 ** -9 * want.norm()


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("gate", [None, "head", "element"])
def test_latent_attention(step, gate):
    from krasis_b200.mixers import WindowLatentAttention
    W, H, R = 256, 4, 128
    g = torch.Generator().manual_seed(6)
    r = lambda *s, sd=W ** -0.5: (torch.randn(*s, generator=g) * sd).bfloat16()  # noqa: E731
    w = {"q": r(H * 192, W), "dkv": r(R + 64, W), "dkv_norm": 1 + r(R, sd=0.1), "uk": r(H * 128, R, sd=R ** -0.5), "uv": r(H * 128, R, sd=R ** -0.5),
         "sink": r(H, sd=1.0), "o": r(W, H * 128, sd=(H * 128) ** -0.5)}
    if gate:
        w["g"] = r(H if gate == "head" else H * 128, W)
    m = WindowLatentAttention(w, H, 128, 64, 128, R, 192 ** -0.5, 512, 64, 10000.0, None, 1e-5, torch.bfloat16, "cuda")
    tb, alone, pages = _tables(step)
    ckv, kr = (torch.randn(pages, 64, c, generator=g).bfloat16().cuda() for c in (R, 64))
    h = torch.randn(tb.T, W, generator=g).bfloat16().cuda()
    got = m.forward(h, tb, ckv, kr, 64)
    for (row0, n, _, _), one in zip(tb.layout, alone):
        want = m.forward(h[row0:row0 + n].contiguous(), one, ckv, kr, 64)
        assert (got[row0:row0 + n] - want).norm() <= 2.0 ** -8 * want.norm()      # bf16 heads (and latents up-projected in bf16)
