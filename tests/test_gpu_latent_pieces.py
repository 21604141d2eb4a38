"""Latent attention of few tokens on the plain kernel against fp64: pieces of all lengths around 8, 16 and 32 keys, empty ones behind them, rows that are loaded 16 bytes at
a time and one number at a time, and keys that are not numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE = 16


def _run(r, dr, dn, H, dtype, at, nsplit, window=1 << 30, sink=False, gate=False, off=0, spoil=None, seed=0):
    from krasis_b200 import seqops as ops
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, S = len(at), len(at)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    P = max(at) // PAGE + 1
    ckv, kr = (torch.empty(S * P * PAGE * w + off, device="cuda", dtype=dtype)[off:].view(S * P, PAGE, w) for w in (r, dr))
    ckv.copy_(n(S * P, PAGE, r))
    kr.copy_(n(S * P, PAGE, dr))
    if spoil is not None:
        ckv[spoil // PAGE, spoil % PAGE, r - 1] = float("nan")           # of the first sequence
    q_abs, proj = n(T, H, r), n(T, H * (dn + dr) + 3)
    tb = ops.StepTables([([0], p, i, list(range(i * P, i * P + P))) for i, p in enumerate(at)], "cuda")
    sinks = n(H) if sink else None
    gates = n(T, H) if gate else None
    out = torch.empty(T, H, r, device="cuda")
    acc, ml = torch.full((T, nsplit, H, r), float("nan"), device="cuda"), torch.full((T, nsplit, H, 2), float("nan"), device="cuda")
    scale = (r + dr) ** -0.5
    ops.check(ops.load().kb2_seq_latent_window_attn(
        q_abs.data_ptr(), proj.data_ptr(), proj.stride(0), T, H, dn, dr, r, ckv.data_ptr(), kr.data_ptr(), ops.dt_code(dtype), tb.positions.data_ptr(), tb.seq_of.data_ptr(),
        tb.pages.data_ptr(), tb.max_pages, PAGE, ops._ptr(sinks), scale, window, out.data_ptr(), None, 0, nsplit, acc.data_ptr(), ml.data_ptr(), ops._ptr(gates),
        gates.stride(0) if gate else 0, torch.cuda.current_stream().cuda_stream))
    for t, p in enumerate(at):
        lo = max(0, p - window + 1)
        rows = [x[t * P:t * P + P].reshape(P * PAGE, -1)[lo:p + 1].double() for x in (ckv, kr)]
        q = torch.cat([q_abs[t], proj[t, :H * (dn + dr)].view(H, dn + dr)[:, dn:]], 1).double()
        k = torch.cat(rows, 1)
        s = q @ k.T * scale
        most = (q.abs() @ k.abs().T * scale).max()
        if sink:
            s = torch.cat([s, sinks.double()[:, None]], 1)
        w = torch.softmax(s, 1)[:, :p + 1 - lo]
        f = torch.sigmoid(gates[t].double())[:, None] if gate else 1.0
        want, room = w @ rows[0] * f, w @ rows[0].abs() * f
        if spoil is not None and t == 0 and lo <= spoil <= p:
            assert bool(want.isnan().all()) and bool(out[t].isnan().all())
            continue
        # a score is a sum of D products, which moves a weight and the sum of all; then sums over the keys and the pieces
        bound = (4 * (r + dr) * 2.0 ** -24 * most + (p + 4 * nsplit + 64) * 2.0 ** -24) * room
        assert bool(((out[t].double() - want).abs() <= bound + 1e-30).all()), (t, p, nsplit)
    return out


@pytest.mark.parametrize("nsplit", [1, 2, 5, 64])
@pytest.mark.parametrize("at", [(0, 7, 8), (15, 16, 17), (31, 32, 33), (70, 135, 500), (511, 3, 100)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_pieces(at, nsplit, dtype):
    _run(512, 64, 128, 16, dtype, at, nsplit, sink=True, gate=True)


# rows in units of 16 bytes or not, of bf16 and of fp32; queries one number at a time; more heads than a block takes and fewer; caches that begin off 16 bytes
@pytest.mark.parametrize("r,dr,dn,H,off", [(40, 8, 5, 3, 0), (36, 4, 8, 9, 0), (33, 7, 4, 2, 0), (128, 64, 128, 8, 1), (64, 32, 16, 1, 4), (1032, 24, 8, 5, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("window", [1 << 30, 20])
def test_forms(r, dr, dn, H, off, dtype, window):
    for nsplit in (1, 7):
        _run(r, dr, dn, H, dtype, (9, 40, 77), nsplit, window, off=off, seed=r)


@pytest.mark.parametrize("spoil", [0, 8, 37, 99])
@pytest.mark.parametrize("nsplit", [1, 13, 40])
def test_what_is_not_a_number(spoil, nsplit):
    _run(128, 64, 128, 4, torch.bfloat16, (99, 50, 120), nsplit, spoil=spoil)
