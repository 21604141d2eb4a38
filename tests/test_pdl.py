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


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", open(path).read())


def _first_argument(text, at):
    """The first argument of the call whose parenthesis opens at `at`."""
    depth = 0
    for i in range(at, len(text)):
        c = text[i]
        depth += c in "([{"
        depth -= c in ")]}"
        if (c == "," and depth == 1 and text.count("<", at, i) <= text.count(">", at, i)) or depth == 0:
            return text[at + 1:i].strip()
    raise AssertionError("unbalanced")


def _launched():
    """{kernel: where} of every programmatic launch, those through a variable among them."""
    found = {}
    for name, text in _sources():
        for m in re.finditer(r"(?:launch_pdl|launch_pdl_clusters|cudaLaunchKernelEx)(\()", text):
            ahead = text[:m.start()]
            what = _first_argument(text, m.start(1))
            if what in ("void (*kernel)(P...)",) or name == "pdl.cuh":       # the helper itself
                continue
            if what == "&cfg":
                what = re.match(r"&cfg,\s*(\w+)", text[m.end(1):]).group(1)
            kernels = re.findall(r"\w+_kernel\b", what)
            if not kernels:                                                 # a variable: what it was last set to
                assert re.fullmatch(r"\w+", what), (name, what)
                kernels = re.findall(r"\w+_kernel\b", re.findall(r"auto %s = ([^;]*);" % what, ahead)[-1])
            assert kernels, (name, what)
            found.update({k: name for k in kernels})
    return found


def _bodies():
    out = {}
    for _, text in _sources():
        for m in re.finditer(r"__global__", text):
            k = re.compile(r"(\w+_kernel)\s*\(").search(text, m.end())
            end = _closing(text, k.end() - 1)
            start = text.index("{", end)
            out[k.group(1)] = (text[k.end():end], text[start:_closing(text, start)])
    return out


def _reads_ahead(params, ahead):
    """What a kernel's statements ahead of its wait do that they must not: leave, or touch memory that its parameters lead to."""
    bad = [w for w in ("return", "__ldg", "tma_load", "tma_gather", "bulk_g2s", "bulk_s2g", "atomic", "cp_async", "ld_stream", "->") if w in ahead]
    for p in re.split(r",(?![^<]*>)", params):
        name = re.search(r"(\w+)\s*$", p.strip())
        if name is None:
            continue
        n = name.group(1)
        if "*" in p:
            bad += [n] if re.search(r"\b%s\s*\[|\*\s*%s\b" % (n, n), ahead) else []
        else:
            bad += [n] if re.search(r"\b%s\.\w+\s*\[|[=(,;?:{&|!<>+-]\s*\*\s*%s\.\w+" % (n, n), ahead) else []
    return bad


def test_launched_kernels_wait():
    bodies, launched = _bodies(), _launched()
    assert len(launched) > 80
    for k in ("split_gemm_kernel", "grouped_gemm_kernel", "split_weight_parts_kernel", "portion_rows_kernel", "dense_pair_kernel"):
        assert k in launched, k
    for name in sorted(launched):
        params, body = bodies[name]
        assert len(re.findall(r"pdl_(?:enter|enter_global|wait)\(", body)) == 1, name
        assert not _reads_ahead(params, body[:re.search(r"pdl_(?:enter|enter_global|wait)\(", body).start()]), name


@pytest.mark.parametrize("name", ["split_weight_parts_kernel", "portion_rows_kernel", "split_gemm_kernel", "conv_run_vec_kernel"])
def test_a_kernel_without_its_wait_is_found(name):
    """The check above on kernels whose wait comes after their first access."""
    params, body = _bodies()[name]
    moved = re.sub(r"(?:kb2::)?pdl_(?:enter|enter_global|wait)\([^;]*;", "", body) + "pdl_wait("
    assert _reads_ahead(params, moved[:moved.index("pdl_wait(")])


def _early(body):
    """Whether a kernel lets the next one come up ahead of its own wait, or of a place where some of its blocks may leave without saying so."""
    wait, at = re.search(r"pdl_(?:enter|enter_global|wait)\([^;]*;", body), re.search(r"pdl_trigger\(", body)
    return at.start() < wait.end() or bool(re.sub(r"[\s]|kb2::", "", body[wait.end():at.start()]))


def test_triggers_stand_behind_the_wait():
    """Right behind it: what is launched early waits for the whole of this kernel, which has then waited for all ahead of it."""
    launched, found = _launched(), []
    for name, (_, body) in _bodies().items():
        if "pdl_trigger(" in body:
            assert name in launched and len(re.findall(r"pdl_trigger\(", body)) == 1 and not _early(body), name
            found.append(name)
    assert sorted(found) == ["act_mul_bf16x8_kernel", "delta_step_kernel", "latent_attn_combine_kernel", "residual_norm_vec_kernel", "side_gate_kernel"]


def test_an_early_trigger_is_found():
    body = _bodies()["side_gate_kernel"][1]
    moved = re.sub(r"(?:kb2::)?pdl_trigger\(\);", "", body)
    assert _early("{ kb2::pdl_trigger();" + moved[1:])


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
