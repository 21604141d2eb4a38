"""A row's product does not depend on the rows beside it: within a kernel family every output sums its K products in one order.  And no family is
less exact than fp32 sums where those were promised."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (columns, K): more and fewer column tiles than SMs, K that a cluster shares and K that one CTA keeps, uneven cuts
SHAPES = [(2048, 2048), (2048, 8192), (16384, 1024), (576, 2048), (272, 320), (1024, 576)]


def _data(rows, N, K, dtype=torch.bfloat16, wdtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    return (torch.randn(rows, K, device="cuda", generator=g).to(dtype), (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(wdtype))


def _rows_agree(f, x, counts):
    whole = f(x[:max(counts)].contiguous())
    for m in counts:
        assert torch.equal(f(x[:m].contiguous()), whole[:m]), m
    at = max(counts) // 3
    n = counts[len(counts) // 2]
    if at + n <= max(counts):
        assert torch.equal(f(x[at:at + n].contiguous()), whole[at:at + n])          # and not on the place among them


@pytest.mark.parametrize("N,K", SHAPES)
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_linear(N, K, out_dtype):
    """The projections of the prefill models: bf16 outputs at any number of rows, fp32 outputs up to 255 and from 256 on."""
    from krasis_b200.attention import linear
    x, w = _data(2500, N, K)
    f = lambda a: linear(a, w, out_dtype=out_dtype)  # noqa: E731
    if out_dtype == torch.bfloat16:
        _rows_agree(f, x, (1, 8, 9, 33, 128, 200, 256, 300, 515, 700, 1000, 1500, 2048, 2500))
    else:
        _rows_agree(f, x, (1, 9, 16, 17, 64, 129, 200, 255))
        _rows_agree(f, x, (256, 300, 515, 700, 1000, 1500, 2048, 2500))


@pytest.mark.parametrize("N,K", SHAPES + [(64, 2048), (16, 512)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_lin(N, K, dtype):
    """The serving mixers' products: above the GEMV's 8 rows up to 255 and from 256 on; narrow outputs and fp32 rows at any number above 8."""
    from krasis_b200.mixers import lin
    for wdtype in {dtype, torch.bfloat16}:
        x, w = _data(2100, N, K, dtype, wdtype)
        for out_dtype in (torch.float32, torch.bfloat16):
            f = lambda a: lin(a, w, out_dtype)  # noqa: E731, B023
            if dtype == torch.float32 or N < 256:
                _rows_agree(f, x, (9, 16, 33, 80, 81, 128, 300, 700, 1500, 2100))
            else:
                _rows_agree(f, x, (9, 16, 17, 64, 129, 200, 255))
                _rows_agree(f, x, (256, 300, 515, 1000, 1500, 2100))


@pytest.mark.parametrize("H,N,K", [(16, 512, 128), (16, 128, 512), (3, 144, 192)])
def test_lin_heads(H, N, K):
    from krasis_b200.mixers import lin_heads
    x, w = _data(600, H * N, K, torch.float32)
    x = x.unsqueeze(1).expand(600, H, K) * torch.arange(1, H + 1, device="cuda")[None, :, None]
    w = w.view(H, N, K)
    _rows_agree(lambda a: lin_heads(a, w, torch.empty(a.shape[0], H, N, device="cuda")), x, (9, 16, 33, 80, 128, 300, 600))


# wide outputs that 128 x 256 tiles would be quicker at, and narrow ones; the sums of an fp32 FMA chain are 8.1e-7 off at K = 2048 and 1.6e-6 at 8192
@pytest.mark.parametrize("N,K", [(12352, 2048), (16384, 2048), (32768, 2048), (1024, 8192), (64, 2048)])
@pytest.mark.parametrize("M", [9, 100, 255, 300])
def test_fp32_outputs_are_as_exact_as_fp32_sums(N, K, M):
    from krasis_b200.mixers import lin
    if M >= 256 and N >= 256:
        pytest.skip("one accumulator, as the 128 x 256 tiles have it")
    x, w = _data(M, N, K)
    want = x.double() @ w.double().T
    assert ((lin(x, w, torch.float32).double() - want).norm() / want.norm()).item() < 7e-7
    # a bf16 result: the nearest bf16 numbers of sums that good; 2e-5 of a rounding error is what sums 7e-7 off can add to it
    got, best = lin(x, w, torch.bfloat16).double(), want.float().bfloat16().double()
    assert (got - want).norm() <= (1 + 2e-5) * (best - want).norm()
