"""Capturing a step does not hand the allocator's cache back to the driver, and a failed capture leaves the eager path working."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_capture_keeps_cached_blocks():
    from krasis_b200.graphs import capture
    x = torch.arange(1000, device="cuda", dtype=torch.float32)
    junk = [torch.empty(8 << 20, dtype=torch.uint8, device="cuda") for _ in range(16)]
    del junk
    held = torch.cuda.memory_reserved()
    graph, out = capture(lambda: x * 2 + 1, torch.device("cuda"))
    assert torch.cuda.memory_reserved() >= held
    x.fill_(3.0)
    graph.replay()
    assert (out == 7.0).all()


def test_decode_capture_keeps_cached_blocks(monkeypatch):
    from krasis_b200.scheduler import Scheduler
    from tests import test_gpu_vofelix as V
    model, _ = V.build(V.model_cfg(V.default_layers()), seed=3, page_size=4)
    emptied = []
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: emptied.append(1))
    s = Scheduler(model, max_tokens=64, max_requests=2, cuda_graphs=True)
    for i in range(3):
        s.step([("a", [i], [0]), ("b", [i + 1], [0])])
    assert any(s._graphs.values()) and not emptied


def test_failed_capture_raises_and_device_stays_usable():
    from krasis_b200.graphs import capture
    x = torch.ones(4, device="cuda")

    def step():
        _ = x + 1
        raise ValueError("on the host")
    with pytest.raises(ValueError, match="on the host"):
        capture(step, torch.device("cuda"))
    assert (x + 1).sum().item() == 8.0
