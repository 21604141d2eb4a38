"""fp32 rows against bf16 and fp32 weights on pairs of CTAs: the tiles that a step of many rows takes, against float64 and, bit for bit, against the same rows
in a step of nine, which run on single CTAs."""
import pytest
import torch

from krasis_b200 import mixers

pytestmark = pytest.mark.gpu

# columns that end in the first and in the second CTA of a tile; row tiles of 96 and 128 that are not full; K in one segment, in four and in eight, of uneven
# length; a K that sums in short chunks; two heads
SHAPES = [(700, 4112, 1088, 1), (450, 12304, 576, 1), (2100, 2064, 320, 1), (2000, 272, 2112, 2), (2500, 144, 8256, 1)]


def _product(x, w, dtype=torch.float32):
    out = torch.empty(x.shape[0], w.shape[0], w.shape[1], device="cuda", dtype=dtype)
    assert mixers._lin_f32(x, w, out)
    return out


def _close(got, x, w):
    want = torch.einsum("mgk,gnk->mgn", x.double(), w.double())
    room = 2.0 ** -21 * torch.einsum("mgk,gnk->mgn", x.double().abs(), w.double().abs())      # as in the other tests of parts
    assert ((got.double() - want).abs() <= room).all()


@pytest.mark.parametrize("M,N,K,G", SHAPES)
def test_rows_of_long_steps(M, N, K, G):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, G, K, device="cuda", generator=g)
    w = (torch.randn(G, N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    got = _product(x, w)
    _close(got, x, w)
    assert torch.equal(_product(x[:9].contiguous(), w), got[:9])
    assert torch.equal(_product(x[M - 9:].contiguous(), w), got[M - 9:])
    assert torch.equal(_product(x, w, torch.bfloat16), got.bfloat16())
    wide = w.float()
    assert torch.equal(_product(x, wide)[:9], _product(x[:9].contiguous(), wide))              # (cut along K by the sizes of three parts)
    # low parts that are no zeros: in one CTA's rows of a tile only, and everywhere
    mixed = wide.clone()
    mixed[:, 128:144, K - 1] = torch.randn(G, 16, device="cuda", generator=g)
    for m in (mixed, torch.randn(G, N, K, device="cuda", generator=g) * K ** -0.5):
        got = _product(x, m)
        _close(got, x, m)
        assert torch.equal(_product(x[:9].contiguous(), m), got[:9])


@pytest.mark.parametrize("M,N,K,G", SHAPES[:1] + SHAPES[3:4])
def test_what_is_not_finite(M, N, K, G):
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(M, G, K, device="cuda", generator=g)
    w = (torch.randn(G, N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    x[3, 0, 5], x[M - 1, G - 1, K - 1], x[200, 0, 0] = float("inf"), float("nan"), -float("inf")
    got = _product(x, w)
    want = torch.einsum("mgk,gnk->mgn", x.double(), w.double()).float()
    for test in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(test(got), test(want))
    rows = [i for i in range(M) if i not in (3, 200, M - 1)]
    _close(got[rows], x[rows], w)


# rows of the tiles that the shapes above take, with bf16 and with fp32 weights; a shape for each that takes tiles of 64
TILES = [s + r for s, r in zip(SHAPES, [(96, 96), (128, 128), (96, 96), (128, 128), (96, 96)])] + [(145, 12304, 4096, 1, 64, 0), (193, 4112, 512, 1, 0, 64)]


@pytest.mark.parametrize("M,N,K,G,narrow,wide", TILES)
def test_forms_that_are_compared(M, N, K, G, narrow, wide):
    """The tests of this file compare pairs of CTAs with single ones: steps of M rows run on the former, of nine on the latter."""
    from krasis_b200 import capi
    dev = torch.cuda.current_device()
    if torch.cuda.get_device_properties(dev).multi_processor_count != 148:
        pytest.skip("the tiles are those of 148 SMs")
    rows = capi.load().kb2_linear_f32_pair_rows
    assert (rows(M, N, K, 0, G, dev), rows(M, N, K, 1, G, dev)) == (narrow, wide)
    assert rows(9, N, K, 0, G, dev) == rows(9, N, K, 1, G, dev) == 0


@pytest.mark.parametrize("M,N,K,G,narrow,wide", TILES[len(SHAPES):])
def test_tiles_of_64_rows(M, N, K, G, narrow, wide):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, G, K, device="cuda", generator=g)
    w = torch.randn(G, N, K, device="cuda", generator=g) * K ** -0.5
    for m in [w.bfloat16()] if narrow else [w, w.bfloat16().float()]:
        got = _product(x, m)
        _close(got, x, m)
        assert torch.equal(_product(x[:9].contiguous(), m), got[:9])
        assert torch.equal(_product(x[M - 9:].contiguous(), m), got[M - 9:])
