"""The tensor-core attention at the edges of its tiles: key counts around 64 and 128, windows that start inside a tile, rows that see nothing in one, and maxima
that grow along the keys (every tile rescales the ones before)."""
import pytest
import torch

from krasis_b200 import capi
from krasis_b200.streams import stream_on

pytestmark = pytest.mark.gpu


def _want(q, k, v, past, scale, window):
    """float64 softmax of q [M, H, d] over k [L, H, d], v [L, H, dv]; and the same with |v|."""
    M, L = q.shape[0], k.shape[0]
    s = torch.einsum("mhd,lhd->hml", q.double(), k.double()) * scale
    away = past + torch.arange(M, device="cuda")[:, None] - torch.arange(L, device="cuda")[None]
    p = torch.softmax(s.masked_fill((away < 0) | (away >= window), float("-inf")), -1)
    return torch.einsum("hml,lhd->mhd", p, v.double()), torch.einsum("hml,lhd->mhd", p, v.double().abs())


def _check(got, q, k, v, past, scale, window):
    want, room = _want(q, k, v, past, scale, window)
    # weights are rounded to bf16, by which they are also normalised, and so is the result: 2^-8 of the sum's terms; the scores' fp32 sums
    assert ((got.double() - want).abs() <= 2.0 ** -7 * room + 1e-5).all()


@pytest.mark.parametrize("past,M", [(0, 1), (0, 63), (0, 64), (0, 65), (0, 127), (0, 128), (0, 129), (127, 1), (128, 2), (200, 57), (1000, 130)])
@pytest.mark.parametrize("dv", [128, 256])
@pytest.mark.parametrize("grows", [False, True])
def test_maps(past, M, dv, grows):
    core, H, G = capi.load(), 2, 1
    g = torch.Generator(device="cuda").manual_seed(past + M)
    L = past + M
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    q, k, v = r(M, H, 128).bfloat16(), r(L, G, 128).bfloat16(), r(L, G, dv).bfloat16()
    if grows:
        q = q.abs()
        k = (k.abs() * torch.linspace(0.01, 3.0, L, device="cuda")[:, None, None]).bfloat16()
    dev = torch.cuda.current_device()
    for window in (1 << 30, 64, 100, 1):
        out = torch.empty(M, H, dv, device="cuda")
        capi.check(core.kb2_fmha_maps_slopes(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), M, past, L, H, G, 1, dv, 128 ** -0.5, 0.0, window, None,
                                             None, None, dev, stream_on(dev)))
        _check(out, q, k.expand(L, H, 128), v.expand(L, H, dv), past, 128 ** -0.5, window)


@pytest.mark.parametrize("past,M", [(0, 1), (0, 128), (0, 129), (127, 1), (200, 57), (1000, 130)])
def test_latent(past, M):
    core, H, L = capi.load(), 2, past + M
    g = torch.Generator(device="cuda").manual_seed(past + M)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    q, kn, kr, v = r(M, H, 192), r(L, H, 128), r(L, 64), r(L, H, 128)
    up = torch.cat([kn.reshape(L, -1), v.reshape(L, -1)], 1).contiguous()
    dev = torch.cuda.current_device()
    for window in (1 << 30, 100):
        out = torch.empty(M, H, 128, device="cuda", dtype=torch.bfloat16)
        capi.check(core.kb2_fmha_latent_gated(q.data_ptr(), up.data_ptr(), kr.data_ptr(), out.data_ptr(), M, past, L, H, 192 ** -0.5, window, None, None, 0, dev,
                                              stream_on(dev)))
        _check(out, q, torch.cat([kn, kr[:, None].expand(L, H, 64)], -1), v, past, 192 ** -0.5, window)


@pytest.mark.parametrize("past,M,more", [(0, 1, 90), (0, 64, 1), (0, 63, 200), (60, 4, 1), (64, 64, 64), (100, 28, 9), (130, 62, 1), (1000, 24, 100)])
def test_rows_of_half_tiles(past, M, more):
    """A last tile with keys in its first half alone: the rows that the same queries have where later ones fill it, bit for bit."""
    core, H, G, L = capi.load(), 3, 1, past + M + more
    g = torch.Generator(device="cuda").manual_seed(past + M)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    dev = torch.cuda.current_device()
    q, up, kr = r(M + more, H, 192), r(L, H * 256), r(L, 64)
    q2, k2 = r(M + more, H, 128), r(L, G, 128)
    for window in (1 << 30, 70):
        got = []
        for m in (M, M + more):
            out = torch.empty(m, H, 128, device="cuda", dtype=torch.bfloat16)
            capi.check(core.kb2_fmha_latent_gated(q.data_ptr(), up.data_ptr(), kr.data_ptr(), out.data_ptr(), m, past, past + m, H, 192 ** -0.5, window, None, None, 0, dev,
                                                  stream_on(dev)))
            parts = [out[:M]]
            for dv in (128, 256):
                v = up[:, :dv].contiguous()
                out, lse = torch.empty(m, H, dv, device="cuda"), torch.empty(m, H, device="cuda")
                capi.check(core.kb2_fmha_maps_slopes(q2.data_ptr(), k2.data_ptr(), v.data_ptr(), out.data_ptr(), m, past, past + m, H, G, 1, dv, 128 ** -0.5, 0.0, window,
                                                     None, lse.data_ptr(), None, dev, stream_on(dev)))
                parts += [out[:M], lse[:M]]
            got.append(parts)
        assert all(torch.equal(a, b) and bool(torch.isfinite(a).all()) for a, b in zip(*got))
