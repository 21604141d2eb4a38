"""Expert outputs summed per token, four columns per thread: the same order of fp32 multiply-adds as a loop over the choices."""
import pytest
import torch

from krasis_b200 import seqops as ops

pytestmark = pytest.mark.gpu


# widths around the 1024 columns of a block and one that the scalar form takes, up to eight choices, more, and more than the table of choices holds
@pytest.mark.parametrize("T,top,W,pos,gate", [(1, 1, 4, True, False), (5, 6, 1020, True, True), (3, 8, 1028, False, False), (7, 9, 2048, True, True),
                                              (2, 64, 512, True, False), (2, 65, 512, True, False), (4, 6, 1022, True, True),
                                              # long steps of few choices: a block per token
                                              (512, 1, 1028, True, True), (1024, 4, 36, False, False), (1024, 2, 4, True, True)])
def test_combine(T, top, W, pos, gate):
    E, ident = 16, 3
    g = torch.Generator().manual_seed(W + top)
    ids = torch.randint(-1, E + ident + 1, (T, top), generator=g, dtype=torch.int32)           # -1 and E + ident: nothing
    w = torch.rand(T, top, generator=g)
    rows = torch.randperm(T * top + 5, generator=g)[:T * top].int() if pos else torch.arange(T * top, dtype=torch.int32)
    y, h = torch.randn(T * top + 5, W, generator=g), torch.randn(T, W, generator=g).bfloat16()
    own, sg = torch.randn(T, W, generator=g), torch.randn(T, 3, generator=g)
    c = [t.cuda() for t in (y, rows, ids, w, h, own, sg)]
    out = torch.empty(T, W, device="cuda")
    ops.check(ops.load().kb2_seq_moe_combine(c[0].data_ptr(), c[1].data_ptr() if pos else None, c[2].data_ptr(), c[3].data_ptr(), T, top, E, ident,
                                             c[4].data_ptr(), 1, c[5].data_ptr() if gate else None, out.data_ptr(), W,
                                             c[6].data_ptr() if gate else None, 3, torch.cuda.current_stream().cuda_stream))
    want, size = torch.zeros(T, W, dtype=torch.float64), torch.zeros(T, W, dtype=torch.float64)
    for t in range(T):
        for k in range(top):
            e = int(ids[t, k])
            r = y[rows[t * top + k]] if 0 <= e < E else h[t].float() if E <= e < E + ident else torch.zeros(W)
            want[t] += w[t, k].double() * r.double()
            size[t] += (w[t, k] * r).abs().double()
    if gate:
        s = torch.sigmoid(sg[:, :1].double())
        want += s * own.double()
        size += (s * own).abs()
    # a sum of top + 1 fused multiply-adds: half a unit in the last place each of at most the sum of the magnitudes; the gate within 2^-21 of itself
    assert ((out.cpu().double() - want).abs() <= size * ((top + 1) * 2.0 ** -24 + 2.0 ** -21) + 1e-30).all()
