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
@pytest.mark.parametrize("M,N,K", [(m, n, k) for m in (9, 100, 255) for n, k in ((12352, 2048), (16384, 2048), (32768, 2048), (1024, 8192), (64, 2048))] +
                         [(300, 64, 2048)])
def test_fp32_outputs_are_as_exact_as_fp32_sums(M, N, K):
    from krasis_b200.mixers import lin
    x, w = _data(M, N, K)
    want = x.double() @ w.double().T
    assert ((lin(x, w, torch.float32).double() - want).norm() / want.norm()).item() < 7e-7
    # a bf16 result: the nearest bf16 numbers of sums that good; 2e-5 of a rounding error is what sums 7e-7 off can add to it
    got, best = lin(x, w, torch.bfloat16).double(), want.float().bfloat16().double()
    assert (got - want).norm() <= (1 + 2e-5) * (best - want).norm()


@pytest.mark.parametrize("W,F", [(2048, 1024), (512, 2560), (256, 8192)])
def test_expert_rows_do_not_depend_on_the_step(W, F):
    """Below a mean of 16 rows per expert and from there on, at the depth of a served model (the ring of a tile wraps, several accumulators per tile)."""
    from krasis_b200.mixers import RoutedExperts
    E, top = 8, 2
    g = torch.Generator().manual_seed(F)
    r = lambda *s, sd: (torch.randn(*s, generator=g) * sd).bfloat16()  # noqa: E731
    w = {"router": r(E, W, sd=W ** -0.5)}
    for e in range(E):
        w.update({f"e{e}_gate": r(F, W, sd=W ** -0.5), f"e{e}_up": r(F, W, sd=W ** -0.5), f"e{e}_down": r(W, F, sd=F ** -0.5)})
    mod = RoutedExperts(w, E, 0, top, torch.bfloat16, "cuda", score="softmax", renorm=True)
    h = r(700, W, sd=1.0).cuda()
    ids, wts, _ = mod.route(h)
    for lens in ((9, 20, 40, 63), (64, 100, 112, 150, 168, 200, 224, 230, 256, 700)):      # tiles of 16; 32, 48, 64 and 128
        outs = {}
        for n in lens:
            hn = h[:n].contiguous()
            y, pos = mod._forward_tensor_core(hn, ids[:n].contiguous(), n * top, None)
            outs[n] = y[pos.long()].view(n, top, W)
        for n in lens:
            assert torch.equal(outs[n], outs[lens[-1]][:n]), n
        x, want = h[:lens[-1]].double(), outs[lens[-1]].double()
        for e in range(E):
            tok, j = torch.nonzero(ids[:lens[-1]] == e, as_tuple=True)
            gu = [(x[tok] @ w[f"e{e}_{n}"].cuda().double().T).bfloat16().double() for n in ("gate", "up")]
            a = (torch.nn.functional.silu(gu[0]) * gu[1]).bfloat16().double()
            ref = a @ w[f"e{e}_down"].cuda().double().T
            # as in the other expert tests: a number next to a rounding edge may fall on the other side, one bf16 step of a few of the F terms
            assert ((want[tok, j] - ref).norm(dim=1) <= 2.0 ** -8 * ref.norm(dim=1)).all()


# a direct call with fp32 output: tiles of 16 rows are as exact as fp32 sums at any depth, the others have one accumulator (1.1e-9 of the sum per K)
@pytest.mark.parametrize("tile", [16, 32, 48, 64])
@pytest.mark.parametrize("N,K", [(272, 2048), (144, 8192)])
def test_binned_product(tile, N, K):
    from krasis_b200 import capi
    core = capi.load()
    E, tiles = 3, 7
    x, _ = _data(tile * tiles, 16, K)
    w = (torch.randn(E, N, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(tile)) * K ** -0.5).bfloat16()
    of = torch.tensor([0, 2, 2, 1, 0, 1, 2], dtype=torch.int32, device="cuda")
    n = torch.tensor([tiles - 1], dtype=torch.int32, device="cuda")                        # the last tile does not exist
    out = torch.full((tile * tiles, N), -7.0, device="cuda")
    capi.check(core.kb2_linear_bf16_binned(x.data_ptr(), w.data_ptr(), out.data_ptr(), tile * tiles, N, K, 1, tile, of.data_ptr(), n.data_ptr(), E, 0,
                                           torch.cuda.current_stream().cuda_stream))
    want = torch.einsum("tmk,tnk->tmn", x.view(tiles, tile, K).double(), w[of.long()].double()).view(-1, N)
    last = tile * (tiles - 1)
    assert (out[last:] == -7.0).all()
    err = ((out[:last].double() - want[:last]).norm() / want[:last].norm()).item()
    assert err < (7e-7 if tile == 16 else 1.2e-9 * K), err
