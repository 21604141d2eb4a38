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


# mean rows per expert on both sides of every tile size (16, 32, 48, 64, 128), with experts that get no row and one that gets most
@pytest.mark.parametrize("T,E,top", [(9, 64, 2), (13, 2, 2), (30, 2, 1), (84, 2, 1), (85, 2, 1), (112, 2, 1), (113, 2, 1), (300, 3, 2), (1500, 5, 3)])
@pytest.mark.parametrize("skew", [0.0, 3.0])
def test_binned_experts_of_any_run_length(T, E, top, skew):
    from krasis_b200.mixers import RoutedExperts
    W, F = 192, 128
    g = torch.Generator().manual_seed(T + E)
    r = lambda *s, sd: (torch.randn(*s, generator=g) * sd).bfloat16()  # noqa: E731
    w = {"router": r(E, W, sd=W ** -0.5)}
    for e in range(E):
        w.update({f"e{e}_gate": r(F, W, sd=W ** -0.5), f"e{e}_up": r(F, W, sd=W ** -0.5), f"e{e}_down": r(W, F, sd=F ** -0.5)})
    bias = torch.zeros(E)
    bias[0] = skew                                            # most rows choose expert 0; with many experts some get none
    w["router_b"] = bias
    h = r(T, W, sd=1.0).cuda()
    mod = RoutedExperts(w, E, 0, top, torch.bfloat16, "cuda", score="softmax")
    assert mod._tensor_core_ok(h, T * top)
    ids, wts, _ = mod.route(h)
    got = mod.forward(h).double().cpu()
    x, want = h.double().cpu(), torch.zeros(T, W, dtype=torch.float64)
    for e in range(E):
        tok, j = torch.nonzero(ids.cpu() == e, as_tuple=True)
        if tok.numel():
            gu = [(x[tok] @ w[f"e{e}_{n}"].double().T).bfloat16().double() for n in ("gate", "up")]
            a = (torch.nn.functional.silu(gu[0]) * gu[1]).bfloat16().double()
            want.index_add_(0, tok, (a @ w[f"e{e}_down"].double().T) * wts.cpu()[tok, j].double()[:, None])
    # the oracle rounds to bf16 where the kernels do; a gate, up or activation next to a rounding edge may fall on the other side: one
    # bf16 step (2^-8) of a few of the F terms, well inside 2^-8 of the row's norm
    assert ((got - want).norm(dim=1) <= 2.0 ** -8 * want.norm(dim=1) + 1e-6).all()


def test_long_and_short_binning_agree():
    """Steps of up to 8192 slots bin in one block, longer ones in three launches: the same tables but for the order inside a run."""
    from krasis_b200.mixers import RoutedExperts
    E = 37
    mod = RoutedExperts({"router": torch.zeros(E, 64), **{f"e{e}_{n}": torch.zeros(64, 64) for e in range(E) for n in ("gate", "up", "down")}}, E, 0, 1,
                        torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    for slots in (1, 8192, 8193, 20000):
        ids = torch.randint(-1, E + 2, (slots,), device="cuda", generator=g, dtype=torch.int32)     # some slots name no expert
        for tile in (16, 64, 128):
            t = mod._bin(ids, slots, tile)
            counts = torch.bincount(ids[(ids >= 0) & (ids < E)].long(), minlength=E)
            tiles = (counts + tile - 1) // tile
            n = int(tiles.sum())
            assert int(t["n_tiles"][0]) == n and torch.equal(t["offs"].long(), torch.cat([tiles.new_zeros(1), tiles.cumsum(0)]) * tile)
            assert torch.equal(t["tile_expert"][:n].long(), torch.arange(E, device="cuda").repeat_interleave(tiles))
            rows = t["slot_row"][:n * tile].long()
            real = rows >= 0
            assert torch.equal(torch.sort(rows[real])[0], torch.nonzero((ids >= 0) & (ids < E)).flatten())
            assert torch.equal(ids[rows[real]].long(), t["tile_expert"][:n].long().repeat_interleave(tile)[real])
            assert torch.equal(t["pos"].long()[rows[real]], torch.nonzero(real).flatten()) and int((t["pos"] < 0).sum()) == slots - int(real.sum())


def _f32(x, w, out):
    from krasis_b200.mixers import _lin_f32
    assert _lin_f32(x, w, out)
    return out


# rows around a tile (16, 80 per tile of parts), uneven K cuts, heads side by side, a slice border of the weight parts (N 8192, K 4096)
@pytest.mark.parametrize("M,N,K,G", [(9, 16, 128, 1), (17, 144, 192, 3), (80, 272, 512, 1), (81, 128, 576, 2), (255, 512, 128, 16), (300, 2048, 2048, 1),
                                     (33, 8192, 4096, 1)])
@pytest.mark.parametrize("wide", [True, False])
def test_fp32_rows_are_as_exact_as_fp32_sums(M, N, K, G, wide):
    from krasis_b200 import seqops as ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, G, K, device="cuda", generator=g) * torch.exp(torch.randn(M, G, 1, device="cuda", generator=g) * 8)      # rows of any size
    w = torch.randn(G, N, K, device="cuda", generator=g) * K ** -0.5
    w = w if wide else w.bfloat16()
    want = torch.einsum("mgk,gnk->mgn", x.double(), w.double())
    err = lambda y: ((y.double() - want).norm(dim=2) / want.norm(dim=2)).square().mean().sqrt().item()  # noqa: E731
    got = _f32(x, w, torch.full((M, G, N), float("nan"), device="cuda"))
    fma = ops.gemm_heads(x, w, torch.empty(M, G, N, device="cuda"))
    assert err(got) <= err(fma) < 4e-6
    half = _f32(x, w, torch.empty(M, G, N, device="cuda", dtype=torch.bfloat16))
    assert ((half.double() - want).abs() <= 2.0 ** -8 * want.abs() + 4e-6 * want.norm(dim=2, keepdim=True)).all()


@pytest.mark.parametrize("wide", [True, False])
def test_fp32_rows_with_extreme_values(wide):
    """Infinities, NaN, the largest and the smallest numbers come out as a plain fp32 product gives them."""
    M, N, K = 24, 128, 128
    g = torch.Generator(device="cuda").manual_seed(2)
    x, w = torch.randn(M, 1, K, device="cuda", generator=g), torch.randn(1, N, K, device="cuda", generator=g)
    x[0, 0, 3], x[1, 0, 5], x[2, 0, 7] = float("inf"), float("-inf"), float("nan")
    x[3], x[4] = 0.0, 0.0
    x[3, 0, 9] = 3.4028e38                       # rounds to infinity in bf16
    x[4, 0, 9] = 1e-38
    x[5, 0, 0], x[5, 0, 1] = float("inf"), float("-inf")
    w = w.bfloat16().float()
    w[0, 7, 3], w[0, 9, :] = 0.0, 0.0            # infinity times zero
    w[0, :, 9] = w[0, :, 9].clamp(-0.875, 0.875)
    if wide:
        w[0, 11, 0] = float("inf")
    want = (x[:, 0].unsqueeze(1).double() * w[0].unsqueeze(0).double()).float().sum(-1)
    got = _f32(x, w if wide else w.bfloat16(), torch.empty(M, 1, N, device="cuda"))[:, 0]
    same = (got == want) | (got.isnan() & want.isnan())
    # beside the rounding of sums: bf16 numbers end at 2^-133, so what a part of x misses is at most 2^-134 in absolute terms, times |w| (it
    # shows for x below 1e-33 only, here in row 4)
    room = 1e-6 * (x[:, 0].abs().unsqueeze(1) * w[0].abs().unsqueeze(0)).sum(-1) + 2.0 ** -133 * w[0].abs().amax(-1)
    assert (same | (want.isfinite() & got.isfinite() & ((got - want).abs() <= room))).all()
