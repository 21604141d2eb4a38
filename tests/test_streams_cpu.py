"""Stream handles: a tensor or device that is not on a GPU is refused before anything is launched on its addresses."""
import pytest
import torch

from krasis_b200 import mixers, streams


@pytest.fixture(autouse=True)
def _runtime(monkeypatch):
    monkeypatch.setattr(streams, "_raw", lambda index: 1000 + index)          # torch's own takes -1 as the current device
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)


def test_handles():
    assert streams.stream_on(2) == 1002 and streams.stream_on("cuda:1") == 1001 and streams.stream_on(torch.device("cuda", 0)) == 1000
    assert streams.stream_on(None) == 1003 and streams.stream_on("cuda") == 1003


@pytest.mark.parametrize("device", ["cpu", torch.device("cpu"), "meta", -1])
def test_other_devices_are_refused(device):
    with pytest.raises(ValueError):
        streams.stream_on(device)


def test_other_tensors_are_refused():
    for t in (torch.zeros(4), torch.zeros(4, device="meta")):
        with pytest.raises(ValueError):
            streams.stream_of(t)


@pytest.mark.parametrize("M", [9, 300])
def test_products_of_host_tensors(M, monkeypatch):
    """lin and lin_glu look at sizes first; the launch itself must not be reached."""
    class Core:
        def __getattr__(self, name):
            if name == "kb2_linear_glu_bf16_takes":
                return lambda *a: 1
            return lambda *a: pytest.fail(f"{name} was called with host addresses")
    monkeypatch.setattr(mixers, "_core", Core())
    monkeypatch.setattr(mixers, "_core_check", lambda rc: None)
    a, w = torch.zeros(M, 128, dtype=torch.bfloat16), torch.zeros(256, 128, dtype=torch.bfloat16)
    for call in (lambda: mixers.lin(a, w), lambda: mixers.lin_glu(a, w, 1, 0.0, 0.0), lambda: mixers.lin(a.float(), w.float())):
        with pytest.raises(ValueError):
            call()
