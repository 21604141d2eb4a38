"""Calls of different shapes from several threads at once."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_delta_tiles_of_different_heads():
    """Heads per key head set the shared memory of the preparation: two threads whose layers differ in them, each on a stream of its own."""
    from krasis_b200 import seqops as ops
    lib, bad = ops.load(), []
    dk = dv = 128
    T = 64

    def work(H, Hk, seed):
        try:
            g = torch.Generator(device="cuda").manual_seed(seed)
            stream = torch.cuda.Stream()
            conv, proj = torch.randn(T, 2 * Hk * dk + H * dv, device="cuda", generator=g), torch.randn(T, H * dv + 2 * H, device="cuda", generator=g)
            A, b, nw = torch.zeros(H, device="cuda"), torch.zeros(H, device="cuda"), torch.ones(dv, device="cuda")
            cu, slots = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
            state, out = torch.zeros(1, H, dk, dv, device="cuda"), torch.empty(T, H * dv, device="cuda")
            size = int(lib.kb2_seq_delta_tiles_scratch(T, 1, H, Hk, dk, dv))
            scratch = torch.empty(size, device="cuda")
            torch.cuda.synchronize()
            first = None
            for i in range(300):
                with torch.cuda.stream(stream):
                    state.zero_()
                    ops.check(lib.kb2_seq_delta_tiles(conv.data_ptr(), conv.shape[1], proj.data_ptr(), proj.stride(0), 0, H * dv, H * dv + H, T, 1, H, Hk, dk,
                                                      dv, A.data_ptr(), b.data_ptr(), nw.data_ptr(), 1e-5, state.data_ptr(), cu.data_ptr(), slots.data_ptr(),
                                                      scratch.data_ptr(), size, out.data_ptr(), 0, stream.cuda_stream))
                    first = out.clone() if first is None else first
            stream.synchronize()
            assert torch.equal(out, first) and torch.isfinite(out).all()
        except Exception as e:          # noqa: BLE001 — reported by the main thread
            bad.append(e)
    threads = [threading.Thread(target=work, args=a) for a in ((2, 2, 0), (32, 2, 1))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
