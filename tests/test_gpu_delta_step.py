"""Steps in which every sequence has one token: the one-launch form of the delta mixer gives what the five launches of other steps give, bit for bit."""
import pytest
import torch

from krasis_b200 import seqops
from krasis_b200.mixers import GatedDeltaMixer

pytestmark = pytest.mark.gpu


# one, two and three heads per key head (the last pair is half empty), two to four taps
@pytest.mark.parametrize("H,Hk,K", [(4, 4, 4), (8, 4, 4), (6, 2, 3), (2, 2, 2), (32, 16, 4)])
@pytest.mark.parametrize("T", [1, 5])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_same_as_separate_launches(H, Hk, K, T, dtype):
    g = torch.Generator().manual_seed(H + K + T)
    W, n, slots = 256, 128, 8
    r = lambda *s, sd=1.0: torch.randn(*s, generator=g) * sd  # noqa: E731
    w = {"g": r(H * n, W, sd=W ** -0.5), "a": r(H, W, sd=W ** -0.5), "b": r(H, W, sd=W ** -0.5), "A_log": r(H), "dt_bias": r(H) - 3.0,
         "norm": 1.0 + 0.1 * r(n), "o": r(W, H * n, sd=(H * n) ** -0.5)}
    for nm, rows in (("q", Hk * n), ("k", Hk * n), ("v", H * n)):
        w[nm], w[nm + "_conv"] = r(rows, W, sd=W ** -0.5), r(rows, K, sd=0.5)
    m = GatedDeltaMixer(w, H, Hk, n, n, K, 1e-5, dtype, "cuda")
    order = [5, 0, 7, 2, 3][:T]
    x = r(3, T, W).cuda().to(dtype)
    ends = []
    for one in (True, False):
        assert m.one_launch
        m.one_launch = one
        tail, state = r(slots, m.C, K - 1).cuda() * 0 + 0.3, torch.full((slots, H, n, n), 0.01, device="cuda")
        outs = [m.forward(x[i], seqops.StepTables([([0], i, s, [0]) for s in order], "cuda"), tail, state) for i in range(3)]
        ends.append(outs + [tail, state])
        m.one_launch = True
    for a, b in zip(*ends):
        assert torch.equal(a, b)
    assert torch.isfinite(ends[0][0]).all()
    untouched = [s for s in range(slots) if s not in order]
    assert (ends[0][-1][untouched] == 0.01).all() and (ends[0][-2][untouched] == 0.3).all()


@pytest.mark.parametrize("H,Hk,K", [(10, 2, 4), (8, 1, 2), (14, 2, 3), (16, 2, 4)])
def test_clusters_of_more_heads(H, Hk, K):
    """Five, seven and eight heads per key head: a cluster of as many blocks."""
    test_same_as_separate_launches(H, Hk, K, 5, torch.bfloat16)


@pytest.mark.parametrize("kw", [{"dk": 64}, {"dv": 64}, {"K": 5}, {"K": 1}, {"H": 18, "Hk": 2}, {"H": 5, "Hk": 2}, {"ldp": 4098}, {"g_off": 2}, {"T": 0}, {"state": 8}])
def test_what_is_refused(kw):
    a = dict(ldp=4096, g_off=1024, T=1, H=4, Hk=2, dk=128, dv=128, K=4, state=0)
    a.update(kw)
    buf = torch.zeros(4, dtype=torch.int32, device="cuda")
    p = buf.data_ptr()
    rc = seqops.load().kb2_seq_delta_step(p, a["ldp"], a["g_off"], 0, 0, a["T"], a["H"], a["Hk"], a["dk"], a["dv"], a["K"], p, p, p, p, p, 1e-5, p + a["state"], p, p, 1, None)
    assert rc == 2


def test_state_off_16_bytes():
    """States that begin off 16 bytes are taken, and give the same bits."""
    g = torch.Generator().manual_seed(2)
    W, n, H, slots = 256, 128, 2, 3
    r = lambda *s, sd=0.06: torch.randn(*s, generator=g) * sd  # noqa: E731
    w = {"g": r(H * n, W), "a": r(H, W), "b": r(H, W), "A_log": r(H), "dt_bias": r(H) - 3.0, "norm": 1.0 + r(n), "o": r(W, H * n)}
    for nm in ("q", "k", "v"):
        w[nm], w[nm + "_conv"] = r(H * n, W), r(H * n, 4, sd=0.5)
    m = GatedDeltaMixer(w, H, H, n, n, 4, 1e-5, torch.bfloat16, "cuda")
    x, tb = r(2, W, sd=1.0).cuda().bfloat16(), seqops.StepTables([([0], 4, 2, [0]), ([0], 9, 0, [0])], "cuda")
    ends = []
    for off in (0, 1):
        state = torch.empty(slots * H * n * n + off, device="cuda")[off:].view(slots, H, n, n).fill_(0.01)
        tail = torch.full((slots, m.C, 3), 0.3, device="cuda")
        ends.append([m.forward(x, tb, tail, state), tail, state])
    for a, b in zip(*ends):
        assert torch.equal(a, b)
