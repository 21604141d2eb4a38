"""The operands of a portion's attention: what the one-launch form does not take is refused or gathered as it was before there was one."""
import types

import pytest
import torch

from krasis_b200 import seqops as ops

PAGE, PAGES = 16, [5, 0, 3, 7]


def _step(n, start, pages=PAGES):
    return types.SimpleNamespace(layout=[(0, 1, 0, [9]), (1, n, start, list(pages))], max_pages=len(pages), pages=torch.zeros(8, dtype=torch.int32))


@pytest.fixture(autouse=True)
def _no_launch(monkeypatch):
    monkeypatch.setattr(ops, "load", lambda: pytest.fail("a kernel would have been launched"))


def _cache(width, form):
    if form == "offset":                       # rows that begin off 16 bytes
        return torch.randn(8 * PAGE * width + 1).bfloat16()[1:].view(8, PAGE, width)
    if form == "strided":                      # a view of wider rows
        return torch.randn(8, PAGE, width + 8).bfloat16()[:, :, :width]
    return torch.randn(8, PAGE, width).to(torch.float32 if form == "fp32" else torch.bfloat16)


@pytest.mark.parametrize("a,b", [("offset", "plain"), ("plain", "offset"), ("strided", "plain"), ("offset", "strided"), ("fp32", "plain")])
@pytest.mark.parametrize("start,n,first", [(0, 1, 0), (20, 30, 3), (16, 48, 16)])
def test_other_caches_are_gathered(a, b, start, n, first):
    wa, wb, nq = 24, 8, 40
    ca, cb, proj = _cache(wa, a), _cache(wb, b), torch.randn(n + 2, nq + 3)
    got = ops.portion_rows(_step(n, start), 1, first, ca, wa, cb, wb, PAGE, proj, 1, n, nq)
    at = [(PAGES[j // PAGE], j % PAGE) for j in range(first, start + n)]
    for c, g in ((ca, got[0]), (cb, got[1])):
        assert torch.equal(g, torch.stack([c[p, r] for p, r in at])) and g.is_contiguous()
    assert torch.equal(got[2], proj[1:1 + n, :nq].bfloat16()) and got[2].is_contiguous()


def test_caches_without_rows_are_refused():
    pair = torch.randn(8, 2, PAGE, 8).bfloat16()                       # keys and values of a page side by side: pages are not rows one after the other
    with pytest.raises(RuntimeError):
        ops.portion_rows(_step(4, 0), 1, 0, pair[:, 0], 8, pair[:, 1], 8, PAGE, torch.randn(6, 8), 1, 4, 8)


@pytest.mark.parametrize("start,n", [(0, 65), (60, 5), (64, 1)])
def test_positions_without_a_page_are_refused(start, n):
    c = torch.randn(8, PAGE, 8).bfloat16()
    with pytest.raises(IndexError):
        ops.portion_rows(_step(n, start), 1, 0, c, 8, c, 8, PAGE, torch.randn(n + 1, 8), 1, n, 8)
