"""Pieces of an attention row put together by strips of 32 columns, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,dv,pieces", [(1, 1, 1, 2), (3, 5, 31, 31), (2, 4, 33, 32), (3, 32, 128, 33), (1, 7, 130, 64), (5, 3, 256, 65), (1, 2, 512, 3)])
@pytest.mark.parametrize("gate", [None, "head", "element"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_merge(T, H, dv, pieces, gate, dtype):
    from krasis_b200 import seqops as ops
    g = torch.Generator(device="cuda").manual_seed(dv + pieces)
    rows = T * H
    acc = torch.randn(rows, pieces, dv, device="cuda", generator=g)
    ml = torch.empty(rows, pieces, 2, device="cuda")
    ml[..., 0] = torch.randn(rows, pieces, device="cuda", generator=g) * 3
    ml[..., 1] = torch.rand(rows, pieces, device="cuda", generator=g) * 30 + 1
    ml[:, 1::3, 0] = -float("inf")                           # pieces without a key
    ml[:, 1::3, 1] = 0
    acc[:, 1::3] = 0
    gates = None if gate is None else torch.randn(T, H if gate == "head" else H * dv, device="cuda", generator=g)
    out = torch.empty(T, H * dv, device="cuda", dtype=dtype)
    ops.check(ops.load().kb2_seq_attn_finish(None, acc.data_ptr(), ml.data_ptr(), pieces, T, H, 1, dv, None, 0, 1e-6, 1.0, ops._ptr(gates),
                                             gates.stride(0) if gates is not None else 0, out.data_ptr(), ops.dt_code(dtype), None, None, 0, int(gate == "element"),
                                             None, None, 0, torch.cuda.current_stream().cuda_stream))
    m, l = ml[..., 0].double(), ml[..., 1].double()
    e = torch.exp(m - m.max(1, keepdim=True).values)
    w = e / (e * l).sum(1, keepdim=True)
    want = torch.einsum("rp,rpd->rd", w, acc.double())
    size = torch.einsum("rp,rpd->rd", w, acc.double().abs())
    s = 1.0
    if gates is not None:
        s = torch.sigmoid(gates.double())
        s = s.reshape(rows, 1) if gate == "head" else s.reshape(rows, dv)
    # exponentials of differences of up to 24 (2^-19.4 of their size), sums and products of `pieces` numbers; then the result's own rounding
    bound = (2.0 ** -19 + (2 * pieces + 8) * 2.0 ** -24) * size * s + (2.0 ** -8 if dtype is torch.bfloat16 else 0.0) * (want * s).abs()
    assert ((out.double().view(rows, dv) - want * s).abs() <= bound).all()
