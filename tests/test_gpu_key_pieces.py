"""The keys of decoded tokens are cut by the room of the page lists: a step replayed from a graph that was captured at a shorter context gives the bits of one that runs
by itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(kind, dtype):
    from krasis_b200.mixers import MultiMapAttention, WindowLatentAttention
    g = torch.Generator().manual_seed(7)
    r = lambda *s: torch.randn(*s, generator=g) * s[-1] ** -0.5  # noqa: E731
    W, H, G, d = 256, 4, 2, 128
    if kind == "latent":
        w = {"q": r(H * 192, W), "dkv": r(128 + 64, W), "dkv_norm": torch.ones(128), "uk": r(H * 128, 128), "uv": r(H * 128, 128), "o": r(W, H * 128)}
        return WindowLatentAttention(w, H, 128, 64, 128, 128, 192 ** -0.5, None, 64, 10000.0, None, 1e-5, dtype, "cuda"), (128, 64)
    maps = 2 if kind == "maps" else 1
    w = {"q": r(H * maps * d, W), "k": r(G * maps * d, W), "v": r(G * d, W), "o": r(W, H * d)}
    kw = {}
    if kind == "gate":
        w["g"] = r(H, W)
    if kind == "chunk":
        kw["chunk"] = 300
    if kind == "window":
        kw["window"] = 200
    if kind == "maps":
        kw["map_coef"], kw["unit_norm"] = [1.0, -0.3], True
    return MultiMapAttention(w, H, G, maps, d, d, d ** -0.5, 1e-5, dtype, "cuda", rot_dims=64, **kw), (G * maps * d, G * d)


@pytest.mark.parametrize("kind", ["plain", "gate", "chunk", "window", "maps", "latent"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_replayed_steps(kind, dtype):
    from krasis_b200 import seqops as ops
    from krasis_b200.graphs import capture
    m, (ka, kb) = _layer(kind, dtype)
    S, P = 2, 8
    g = torch.Generator(device="cuda").manual_seed(1)
    kc, vc = (torch.randn(S * P, 64, c, device="cuda", generator=g).to(dtype) for c in (ka, kb))
    h = torch.randn(S, 256, device="cuda", generator=g).to(dtype)

    def entries(past):
        return [([0], p, i, list(range(i * P, i * P + p // 64 + 1))) for i, p in enumerate(past)]
    buf = torch.zeros(3 * S + S + 1 + S + S * P, dtype=torch.int32, device="cuda")
    tb = ops.StepTables(entries((5, 21)), "cuda", pad_pages_to=8, device_buf=buf)
    k1, v1 = kc.clone(), vc.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        m.forward(h, tb, k1, v1, 64)
    torch.cuda.current_stream().wait_stream(side)
    graph, out = capture(lambda: m.forward(h, tb, k1, v1, 64), "cuda")
    for past in ((5, 21), (40, 130), (420, 97), (511, 0)):
        k1.copy_(kc)
        v1.copy_(vc)
        k2, v2 = kc.clone(), vc.clone()
        ops.StepTables(entries(past), "cuda", pad_pages_to=8, device_buf=buf)
        graph.replay()
        want = m.forward(h, ops.StepTables(entries(past), "cuda"), k2, v2, 64)
        assert torch.equal(out, want) and torch.equal(k1, k2) and torch.equal(v1, v2) and bool(torch.isfinite(want).all())
