"""Programmatic dependent launches (csrc/pdl.cuh): every kernel that is launched so waits before it touches memory, and chains of such launches
give what the same launches give one at a time."""
import glob
import os
import re

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "krasis_b200", "csrc")


def _closing(text, at):
    depth = 0
    for i in range(at, len(text)):
        depth += {"(": 1, ")": -1, "{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def test_launched_kernels_wait():
    bodies, launched = {}, set()
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            k = re.compile(r"(\w+_kernel)\s*\(").search(text, m.end())
            start = text.index("{", _closing(text, k.end() - 1))
            bodies[k.group(1)] = text[start:_closing(text, start)]
        launched |= set(re.findall(r"launch_pdl\((\w+_kernel)", text))
    launched |= {"split_gemm_kernel", "grouped_gemm_kernel"}               # launched through a variable
    assert len(launched) > 60
    for name in sorted(launched):
        calls = re.findall(r"pdl_(?:enter|wait)\(", bodies[name])
        assert len(calls) == 1, name
        ahead = bodies[name][:re.search(r"pdl_(?:enter|wait)\(", bodies[name]).start()]
        assert "return" not in ahead and "__ldg" not in ahead and "tma_load" not in ahead and "bulk_g2s" not in ahead, name


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 8, 77, 300])
def test_chain_equals_single_launches(rows):
    """Inputs and weights are rewritten right ahead of the kernels that read them, in buffers that earlier kernels have read."""
    from krasis_b200 import seqops as ops
    from krasis_b200.mixers import lin
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = [torch.randn(512, 512, device="cuda", generator=g).mul_(512 ** -0.5).bfloat16() for _ in range(3)]
    x0 = torch.randn(rows, 512, device="cuda", generator=g)
    wn = torch.ones(512, device="cuda")

    def chain(sync):
        x, h, wt = x0.clone(), torch.empty(rows, 512, dtype=torch.bfloat16, device="cuda"), torch.empty_like(w[0])
        for i in range(30):
            wt.copy_(w[i % 3])
            h = ops.residual_add_norm(x, out_norm=(wn, None), out_dtype=torch.bfloat16)
            sync()
            y = lin(h, wt, torch.float32)
            sync()
            h = ops.residual_add_norm(x, y, out_norm=(wn, None), out_dtype=torch.bfloat16)
            sync()
            y = lin(h, wt, torch.float32)
            wt.zero_()
            sync()
            x = ops.residual_add_norm(x, y, out_norm=(wn, None), out_dtype=torch.float32)
            sync()
        return x
    assert torch.equal(chain(lambda: None), chain(torch.cuda.synchronize))
