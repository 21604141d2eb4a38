"""SiLU of the sequence operators at its ends and against fp64, through a convolution that passes its input on."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [3, 96])                       # a thread per number, and four channels by sixteen rows
def test_silu(T):
    from krasis_b200 import seqops as ops
    g = torch.Generator(device="cuda").manual_seed(T)
    C = 2048
    x = torch.randn(T, C, device="cuda", generator=g) * torch.logspace(-42, 37, C, device="cuda")
    ends = torch.tensor([0.0, -0.0, 1e-45, -1e-45, 3.4e38, -3.4e38, -86.5, -87.5, -88.0, -88.5, -88.8, -103.0, float("inf"), -float("inf"), float("nan")], device="cuda")
    x[0, :ends.numel()] = ends
    x[1] = torch.linspace(-100.0, 30.0, C, device="cuda")
    x[2] = torch.linspace(-4.0, 4.0, C, device="cuda")
    taps = torch.tensor([0.0, 1.0], device="cuda").repeat(C, 1)
    # the tap of 0 would turn an infinity of the row ahead into NaN: only row 0 holds some, and row 1 leaves their channels out
    tb = ops.StepTables([([0] * T, 0, 0, [0])], "cuda")
    got = ops.conv(x, C, taps, None, True, torch.zeros(1, C, 1, device="cuda"), tb).double()
    z = x.double()
    want = z / (1.0 + torch.exp(-z))
    odd = ~torch.isfinite(x)
    odd[1] |= odd[0]
    # expf 2 ulp (2^-22), a sum (2^-24), a quotient (2^-23); where e^-x passes fp32's largest number the answer is 0 for at most 89 e^-88.7
    assert ((got - want).abs() <= 2.0 ** -21 * want.abs() + 3e-37)[~odd].all()
    i = ends.numel()
    assert got[0, i - 3] == float("inf") and got[0, i - 2:i].isnan().all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sign_of_zero(dtype):
    """silu(-0) u is -0 u, and so is a clamped swish of it."""
    from krasis_b200 import seqops as ops
    F = 64
    g = torch.zeros(2, F, device="cuda")
    g[:, ::2] = -0.0
    gu = torch.cat([g, torch.ones(2, F, device="cuda")], 1).to(dtype)
    for kind, kw in ((1, {}), (2, {"limit": 7.0, "alpha": 1.7})):
        got = ops.glu(gu, dtype, kind, **kw)
        assert torch.equal(got.float().signbit(), g.signbit()) and not got.any()


def _arguments(n):
    """Numbers of either sign and all sizes, a fine row around zero, and both ends of exp."""
    size = torch.logspace(-44, 38, n // 4, device="cuda")
    return torch.cat([size, -size, torch.linspace(-4.0, 4.0, n // 4, device="cuda"), torch.linspace(-104.0, 104.0, n - 3 * (n // 4), device="cuda")])


@pytest.mark.parametrize("act", ["silu", "sigmoid"])
@pytest.mark.parametrize("dv", [64, 63])                     # four columns a lane, and one
def test_gates(act, dv):
    from krasis_b200 import seqops as ops
    T, H = 128, 2
    z = _arguments(T * H * dv).view(T, H * dv)
    got = ops.head_norm_gate(torch.ones_like(z), H, dv, torch.float32, gate=z, gate_act=act).double()
    x = z.double()
    want = (x if act == "silu" else 1.0) / (1.0 + torch.exp(-x))
    # expf 2 ulp (2^-22), a sum (2^-24), a quotient (2^-23); where e^-x passes fp32's largest number the answer is 0 for x e^-88.7 or e^-88.7, and what lies below fp32's
    # smallest normal number is rounded to multiples of 2^-149
    assert ((got - want).abs() <= 1.75 * 2.0 ** -22 * want.abs() + (3e-37 if act == "silu" else 4e-39)).all()
    ends = torch.tensor([[float("inf"), -float("inf"), float("nan"), 0.0]], device="cuda").repeat(1, dv)[:, :dv].contiguous()
    got = ops.head_norm_gate(torch.ones_like(ends), 1, dv, torch.float32, gate=ends, gate_act=act)[0, :4].tolist()
    assert got[0] == (float("inf") if act == "silu" else 1.0) and got[2] != got[2] and got[3] == (0.0 if act == "silu" else 0.5)
    assert got[1] != got[1] if act == "silu" else got[1] == 0.0


@pytest.mark.parametrize("F", [4096, 4095])
def test_clamped_swish(F):
    """g' sigmoid(alpha g') (u' + 1) with g' = min(g, limit), u' = clamp(u, -limit, limit)."""
    from krasis_b200 import seqops as ops
    limit, alpha = 7.0, 1.702
    g = torch.stack([_arguments(F), torch.linspace(-60.0, 9.0, F, device="cuda")])
    u = torch.linspace(-9.0, 9.0, F, device="cuda").repeat(2, 1)
    got = ops.glu(torch.cat([g, u], 1).contiguous(), torch.float32, ops.GLU_CLAMPED_SWISH, limit=limit, alpha=alpha).double()
    a = torch.tensor(alpha, device="cuda").double()           # as fp32 has it
    x, y = g.double().clamp(max=limit), u.double().clamp(-limit, limit)
    want = x / (1.0 + torch.exp(-a * x)) * (y + 1.0)
    # as above, the argument of expf rounded once (|alpha x| 2^-24 of e^-alpha x) up to where the answer is 0, u + 1 and the product once each
    room = (1.75 * 2.0 ** -22 + 2.0 ** -23 + (a * x).abs().clamp(max=104.0) * 2.0 ** -24) * want.abs() + 2.0 ** -24 * x.abs() / (1.0 + torch.exp(-a * x))
    assert ((got - want).abs() <= room + 2e-36).all()
