"""Few fp32 rows against bfloat16 weights as three bfloat16 parts: errors of fp32 sums, rows that do not notice one another, and what is not finite."""
import pytest
import torch

from krasis_b200 import seqops as ops

pytestmark = pytest.mark.gpu


# columns around 16 and 32 rows of weights and around the counts that change the split along K; K that ends inside a step, a piece and a warp's turn
@pytest.mark.parametrize("N,K", [(1, 8), (17, 40), (257, 2056), (1000, 64), (4720, 136), (4736, 2048), (9504, 328), (40000, 72),
                                 (257, 4104), (1041, 8200), (300, 16392)])        # two and four blocks along K
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
def test_few_fp32_rows(N, K, out):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    x = torch.randn(8, K, device="cuda", generator=g) * torch.logspace(-12, 12, 8, device="cuda")[:, None]
    got = ops.gemm(x, w, out)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # sums of 32 products that lose up to 2^-23 of their magnitude an instruction, joined in fp32: 2^-20 of the magnitudes is four times that
    assert ((got.double() - want).abs() <= size * 2.0 ** -20 + (want.abs() * 2.0 ** -8 if out is torch.bfloat16 else 0)).all()
    for m in (1, 2, 5):
        assert torch.equal(ops.gemm(x[:m], w, out), got[:m])


@pytest.mark.parametrize("N,K", [(4800, 512), (300, 16392)])
def test_not_finite(N, K):
    g = torch.Generator(device="cuda").manual_seed(0)
    w, x = torch.randn(N, K, device="cuda", generator=g).bfloat16(), torch.randn(4, K, device="cuda", generator=g)
    x[0, 3], x[1, 500] = float("inf"), float("nan")
    w[7, 9] = float("-inf")
    got, want = ops.gemm(x, w, torch.float32), x.double() @ w.double().T
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    inf = torch.isinf(want)
    assert torch.equal(got[inf].sign(), want[inf].sign().float())


def test_a_row_that_is_not_finite_costs_no_more_than_a_few_products():
    """Its sums are made again one after the other, each by a warp: not by one thread along all of K."""
    g = torch.Generator(device="cuda").manual_seed(2)
    w, x = torch.randn(16384, 8192, device="cuda", generator=g).bfloat16(), torch.randn(4, 8192, device="cuda", generator=g)

    def best(x):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ops.gemm(x, w, torch.float32)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    plain = best(x)
    x[2, 77] = float("nan")
    got = ops.gemm(x, w, torch.float32)
    assert torch.isnan(got[2]).all() and torch.isfinite(got[[0, 1, 3]]).all()
    assert best(x) < 8 * plain          # a warp: the weights once more, in turn; a thread reads 2 bytes of them at a time, hundreds of times in turn


# the second and third part of numbers below 1e-33 lie below the smallest bf16 number; the largest numbers have parts that overflow where those are kept
@pytest.mark.parametrize("N,K", [(40, 256), (4800, 64)])
def test_smallest_and_largest_numbers(N, K):
    g = torch.Generator(device="cuda").manual_seed(N)
    w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    scale = torch.tensor([1e-30, 1e-34, 1e-36, 1e-37, 3e-38, 1e-39, 1e35, 1e-45], device="cuda", dtype=torch.float64)
    x = (torch.randn(8, K, device="cuda", generator=g).double() * scale[:, None]).float()
    x[6] = x[6].clamp(-3.4e38 / K, 3.4e38 / K)
    x[6, 3] = 3.4e38                                    # of which the parts overflow, against a weight that leaves the sum finite
    w[:, 3] = 0.25
    got, want = ops.gemm(x, w, torch.float32), x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    # as for other numbers, and K sums and products that end at the smallest fp32 number, 2^-149, each rounded to a multiple of it
    assert ((got.double() - want).abs() <= size * 2.0 ** -20 + K * 2.0 ** -149).all()
