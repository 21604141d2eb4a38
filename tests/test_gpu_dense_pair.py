"""Dense products on pairs of CTAs: the sums of the one-CTA tiles and of the few-row tiles, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows around the pair's 256 and one CTA's 128, columns that end in the first or the second CTA's half of a tile, one K block and many, several rounds
@pytest.mark.parametrize("M,N,K", [(2049, 16, 64), (2304, 272, 128), (2100, 2048, 192), (2500, 3648, 2048), (4481, 1040, 576), (8192, 528, 256),
                                   (2113, 12352, 320), (700, 16384, 256), (1500, 9216, 512)])
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
