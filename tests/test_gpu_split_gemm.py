"""The tensor-core product for few rows (split_gemm.cu) at the edges of its tiles, K cuts and row counts, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bound(x, w):
    """The tensor core adds 16 products to an accumulator at a time and truncates, losing at most 2^-22 of the magnitudes added; sums of 512
    products (32 additions) then meet in round-to-nearest fp32, a handful more additions: 40 * 2^-22 * sum |x||w| covers both."""
    return 40 * 2.0 ** -22 * (x.double().abs() @ w.double().abs().T)


# rows around the tile of 16 and around 256, columns around the tile of 128, K with and without a cut over a cluster and an uneven one
@pytest.mark.parametrize("M,N,K", [(1, 16, 64), (9, 128, 64), (16, 144, 128), (17, 112, 192), (77, 272, 2048), (128, 2048, 576), (255, 240, 1024),
                                   (256, 576, 320), (257, 512, 2048), (515, 2048, 4096), (1000, 64, 2048), (2048, 256, 512)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_few_rows_product(M, N, K, out_dtype):
    from krasis_b200.attention import linear
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    b = torch.randn(N, device="cuda", generator=g)
    for bias in (None, b):
        want = x.double() @ w.double().T + (bias.double() if bias is not None else 0.0)
        got = linear(x, w, bias=bias, out_dtype=out_dtype)
        room = _bound(x, w) + 2.0 ** -23 * want.abs() + (2.0 ** -8 * want.abs() if out_dtype == torch.bfloat16 else 0.0)
        assert ((got.double() - want).abs() <= room).all()
        assert torch.equal(got, linear(x, w, bias=bias, out_dtype=out_dtype))          # sums meet in a fixed order


def test_error_is_that_of_fp32_sums():
    """At K = 8192 the 2-norm error stays at that of an fp32 FMA chain (6e-7 at K = 2048, 1.2e-6 at 8192), where one tensor-core accumulator
    over all of K would be 8e-6 off."""
    from krasis_b200.attention import linear
    g = torch.Generator(device="cuda").manual_seed(3)
    for M in (9, 200):
        x = torch.randn(M, 8192, device="cuda", generator=g).bfloat16()
        w = (torch.randn(1024, 8192, device="cuda", generator=g) * 8192 ** -0.5).bfloat16()
        want = x.double() @ w.double().T
        got = linear(x, w, out_dtype=torch.float32).double()
        assert ((got - want).norm() / want.norm()).item() < 7e-7


def test_misaligned_rows_take_the_general_kernel():
    """A view that starts off a 16-byte boundary cannot be read by TMA; `lin` serves it all the same."""
    from krasis_b200.mixers import lin
    flat = torch.randn(40 * 128 + 1, device="cuda").bfloat16()
    x, w = flat[1:].view(40, 128), torch.randn(48, 128, device="cuda").bfloat16()
    want = x.double() @ w.double().T
    assert ((lin(x, w, torch.float32).double() - want).abs() <= _bound(x, w) + 1e-6).all()
