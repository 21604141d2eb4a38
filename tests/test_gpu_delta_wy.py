"""The delta rule sixteen tokens at a time: value columns in passes, odd numbers of heads per key head, long read-outs, against the rule token by
token and fp64."""
import pytest
import torch

from tests.test_gpu_delta_tiles import _rule

pytestmark = pytest.mark.gpu


# passes of 128 value columns (one, two) and of 32 (five); one, three and five heads per key head, which are taken in pairs; tiles cut short
@pytest.mark.parametrize("H,Hk,dk,dv", [(2, 2, 128, 128), (3, 1, 64, 256), (5, 1, 32, 160), (6, 2, 128, 128)])
@pytest.mark.parametrize("lens", [[15, 1, 16], [33, 47]])
def test_passes_and_pairs(H, Hk, dk, dv, lens):
    g = torch.Generator(device="cuda").manual_seed(H + dv)
    T = sum(lens)
    conv, proj = torch.randn(T, 2 * Hk * dk + H * dv, device="cuda", generator=g), torch.randn(T, H * dv + 2 * H, device="cuda", generator=g)
    state = torch.randn(len(lens), H, dk, dv, device="cuda", generator=g)
    got, got_state = _rule(conv, proj, H, Hk, dk, dv, lens, state)
    want, want_state = _rule(conv, proj, H, Hk, dk, dv, lens, state, tiles=False)
    # both are fp32 sums of some hundred terms in different orders: 16 roundings of 2^-24 in the 2-norm at most (measured 2 to 4)
    assert (got - want).norm() <= 16 * 2.0 ** -24 * want.norm() and (got_state - want_state).norm() <= 16 * 2.0 ** -24 * want_state.norm()


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("T,H", [(592, 32), (1187, 16), (593, 32)])        # 148 * 16 blocks of eight rows: the first length of the four-row form
def test_long_read_out(T, H, dtype):
    """Long steps: each row of the read-out is the row a short step gives, bit for bit."""
    from krasis_b200 import seqops as ops
    g = torch.Generator(device="cuda").manual_seed(T)
    lib, s = ops.load(), torch.cuda.current_stream().cuda_stream
    dk, dv = 32, 128
    conv, proj = torch.randn(T, 2 * dk + H * dv, device="cuda", generator=g), torch.randn(T, H * dv + 2 * H, device="cuda", generator=g)
    A, b, nw = torch.zeros(H, device="cuda"), torch.zeros(H, device="cuda"), torch.rand(dv, device="cuda", generator=g) + 0.5

    def run(rows):
        n = rows.stop - rows.start
        cu, slots = torch.tensor([0, n], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        state = torch.zeros(1, H, dk, dv, device="cuda")
        size = int(lib.kb2_seq_delta_tiles_scratch(n, 1, H, 1, dk, dv))
        scratch, out = torch.empty(size, device="cuda"), torch.empty(n, H * dv, device="cuda", dtype=torch.bfloat16 if dtype else torch.float32)
        c, p = conv[rows].contiguous(), proj[rows].contiguous()
        ops.check(lib.kb2_seq_delta_tiles(c.data_ptr(), c.shape[1], p.data_ptr(), p.stride(0), 0, H * dv, H * dv + H, n, 1, H, 1, dk, dv, A.data_ptr(),
                                          b.data_ptr(), nw.data_ptr(), 1e-5, state.data_ptr(), cu.data_ptr(), slots.data_ptr(), scratch.data_ptr(), size,
                                          out.data_ptr(), dtype, s))
        return out
    whole = run(slice(0, T))
    assert torch.equal(whole[:64], run(slice(0, 64))) and torch.isfinite(whole).all()
