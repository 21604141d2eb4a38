"""GEMV, residual norm and embedding at the sizes where their vector forms begin and end, against fp64 / plain torch."""
import pytest
import torch

from krasis_b200 import seqops as ops

pytestmark = pytest.mark.gpu


# columns around the warp's 16 rows, K around a piece of 128 and its cut over 2, 4, 8 and 16 warps, per-head batches, K off a multiple of 8
@pytest.mark.parametrize("N,K,H", [(1, 8, 1), (15, 120, 1), (17, 136, 3), (100, 256, 1), (1000, 2048, 1), (2049, 4096, 1), (512, 128, 16), (128, 512, 16),
                                   (40000, 256, 1), (33, 100, 1)])
@pytest.mark.parametrize("M", [1, 2, 3, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gemv(N, K, H, M, dtype):
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    a = torch.randn(M, H, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(H, N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    want = torch.einsum("mhk,hnk->mhn", a.double(), w.double())
    # K rounded additions of 2^-24 each at most, of the magnitudes added (far above what a few running sums do); a bf16 result rounds once more
    room = 2.0 ** -24 * min(K, 64) * torch.einsum("mhk,hnk->mhn", a.double().abs(), w.double().abs())
    for out_dtype in (torch.float32, torch.bfloat16):
        got = ops.gemm_heads(a, w, torch.full((M, H, N), float("nan"), device="cuda", dtype=out_dtype))
        assert ((got.double() - want).abs() <= room + (2.0 ** -8 * want.abs() if out_dtype == torch.bfloat16 else 0.0)).all()
    if H == 1:                                    # a row alone is that row of a batch, to the order of the sums
        one = ops.gemm_heads(a[:1], w, torch.empty(1, 1, N, device="cuda"))
        assert ((one[0].double() - want[0]).abs() <= room[0]).all()
    full = ops.gemm_heads(a, w, torch.empty(M, H, N, device="cuda"))
    for m in range(M):                            # and bit for bit, at whatever place
        assert torch.equal(ops.gemm_heads(a[m:m + 1], w, torch.empty(1, H, N, device="cuda"))[0], full[m])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,K", [(8192, 2048), (32768, 2048), (256, 2048), (512, 1024), (128, 8184)])
def test_lin_of_few_rows(N, K, dtype):
    """Up to 8 rows: one form and one order of the sums, and the accuracy of a few running fp32 sums (measured 0.6e-7 to 2.2e-7)."""
    from krasis_b200.mixers import lin
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn(8, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    full, want = lin(a, w, torch.float32), a.double() @ w.double().T
    assert ((full.double() - want).norm() / want.norm()).item() < 3e-7
    for m in (1, 2, 3, 4, 7):
        assert torch.equal(lin(a[:m].contiguous(), w, torch.float32), full[:m]), m


# at the first number, within and at the end of a piece, in the middle and in the last one; K past one piece of every cut
@pytest.mark.parametrize("M", [1, 4, 8])
@pytest.mark.parametrize("N,K", [(512, 2048), (70000, 264), (64, 16392)])
def test_gemv_keeps_infinities(N, K, M):
    """An infinite or overflowing sum is what plain fp32 sums give, infinity and not NaN; the other outputs are as without it."""
    g = torch.Generator(device="cuda").manual_seed(N)
    inf, nan = float("inf"), float("nan")
    a = (torch.randn(M, K, device="cuda", generator=g).abs() + 0.1).bfloat16()          # one sign: no infinities that cancel
    w0 = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    want0 = ops.gemm(a, w0)
    at = sorted({0, 31, 127, 128, K // 2, K - 1})
    for i, values in enumerate([[inf], [-inf], [nan], [inf, -inf], [3e38, 3e38], [-3e38, -3e38]]):
        w = w0.clone()
        rows = torch.arange(len(at), device="cuda") * 9 + i                              # a weight row per place
        for r, k in zip(rows.tolist(), at):
            for j, v in enumerate(values):
                w[r, (k + 200 * j) % K] = v
        big = a.clone()
        if abs(values[0]) < inf:
            big[:] = 1.0                                                                 # two terms of 3e38 overflow
        want = (big.double() @ w[rows].double().T).float()                               # beyond fp32: infinite
        got = ops.gemm(big, w)
        torch.testing.assert_close(got[:, rows], want, rtol=0, atol=0, equal_nan=True)
        if abs(values[0]) == inf:
            keep = torch.ones(N, dtype=torch.bool, device="cuda")
            keep[rows] = False
            assert torch.equal(got[:, keep], want0[:, keep])


@pytest.mark.parametrize("W", [1, 6, 512, 1024, 1028, 2048, 2052, 4096, 4100, 8192, 8196])
@pytest.mark.parametrize("mode", ["layer", "rms", "plain", "none"])
@pytest.mark.parametrize("x0", [False, True])
def test_residual_norm(W, mode, x0):
    g = torch.Generator(device="cuda").manual_seed(W)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    T, eps = 3, 1e-5
    x, y, y2, e0 = r(T, W) * 3, r(T, W) + 1, r(T, W), r(T, W)
    wa, ba, wb, bb = r(W), r(W), r(W), r(W)
    d = lambda t: t.double()  # noqa: E731

    def layer(v, w, b):
        c = v - v.mean(1, keepdim=True)
        return c / torch.sqrt(c.square().mean(1, keepdim=True) + eps) * d(w) + d(b)
    upd = {"layer": lambda: layer(d(y), wa, ba), "plain": lambda: d(y) + d(y2), "none": lambda: 0.0,
           "rms": lambda: d(y) / torch.sqrt(d(y).square().mean(1, keepdim=True) + eps) * d(wa)}[mode]()
    want = d(x) + upd + (d(e0) if x0 and mode != "plain" else 0.0)
    for dt in (torch.float32, torch.bfloat16):
        xs = x.clone()
        if mode == "plain":
            h = ops.residual_add_norm(xs, y, y2, out_norm=(wb, bb), out_dtype=dt, eps=eps)
        else:
            h = ops.residual_norm(xs, y if mode != "none" else None, {"layer": ("layer", wa, ba), "rms": ("rms", wa)}.get(mode), x0=e0 if x0 else None,
                                  out_norm=(wb, bb), out_dtype=dt, eps=eps)
        # fp32 sums of W numbers in a tree, and a handful of operations per element: 2^-20 of the row's largest terms is ample
        assert (xs.double() - want).abs().max() <= 2.0 ** -20 * want.abs().max().clamp_min(1.0) + 2.0 ** -20 * 10
        out = layer(xs.double(), wb, bb)
        assert ((h.double() - out).abs() <= 2.0 ** -18 * (1 + out.abs()) + (2.0 ** -8 * out.abs() if dt == torch.bfloat16 else 0.0)).all()


@pytest.mark.parametrize("W", [4, 8, 12, 2048, 2056, 4104])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embed(W, dtype):
    table = torch.randn(50, W, device="cuda").to(dtype)
    tokens = torch.tensor([0, 49, 7, 7], dtype=torch.int32, device="cuda")
    assert torch.equal(ops.embed(table, tokens, 1.5), table[tokens.long()].float() * 1.5)
    off = torch.randn(50 * W + 1, device="cuda").to(dtype)[1:].view(50, W)          # rows off a 16-byte boundary
    assert torch.equal(ops.embed(off, tokens, 0.5), off[tokens.long()].float() * 0.5)


@pytest.mark.parametrize("T,F,at", [(1, 4, 0), (3, 1028, 0), (5, 8192, 0), (3, 1028, 1), (2, 1027, 0)])
def test_act_mul_of_fp32_rows(T, F, at):
    """Widths in groups of four and not, rows that do not start on 16 bytes: the same numbers from either form."""
    base = torch.randn(T * 2 * F + at, device="cuda", generator=torch.Generator(device="cuda").manual_seed(F))
    gu = base[at:].view(T, 2 * F)
    want = torch.nn.functional.gelu(gu[:, :F].double(), approximate="tanh") * gu[:, F:].double()
    got = ops.act_mul(gu, torch.float32)
    # tanhf and seven products and sums in fp32, of numbers that are 1 + tanh at most twice as large as the result
    assert ((got.double() - want).abs() <= 16 * 2.0 ** -23 * (gu[:, :F].double().abs() * gu[:, F:].double().abs()) + 1e-12).all()
