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
