"""Handles of CUDA streams, for the C interfaces."""
import torch

# The current stream's handle straight from torch's runtime: the Stream object that torch.cuda.current_stream makes on the way costs 2 to 3 us, as
# much as a launch.
_raw = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda index: torch.cuda.current_stream(index).cuda_stream)


def stream_of(t: torch.Tensor) -> int:
    """Handle of the current stream of the CUDA tensor t's device."""
    index = t.get_device()            # negative: not on a GPU
    return _raw(index) if index >= 0 else _refuse(t.device)


def stream_on(device) -> int:
    """Handle of the current stream of a CUDA device (a torch.device, its name or its number; without a number, or for None, the current one)."""
    index = device
    if device is not None and not isinstance(device, int):
        d = torch.device(device)
        if d.type != "cuda":
            _refuse(d)
        index = d.index
    if index is None:
        index = torch.cuda.current_device()
    if index < 0:                     # what a tensor that is not on a GPU gives as its device's number; the runtime would take it as the current one
        _refuse(index)
    return _raw(index)


def _refuse(device):
    """Whoever asks for a stream is about to hand addresses of that device to a kernel."""
    raise ValueError(f"expected a CUDA device, but got {device}")
