"""Handles of CUDA streams, for the C interfaces."""
import torch

# The current stream's handle straight from torch's runtime: the Stream object that torch.cuda.current_stream makes on the way costs 2 to 3 us, as
# much as a launch.
_raw = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda index: torch.cuda.current_stream(index).cuda_stream)


def stream_of(t: torch.Tensor) -> int:
    """Handle of the current stream of the CUDA tensor t's device."""
    return _raw(t.get_device())


def stream_on(device) -> int:
    """Handle of the current stream of a device (a torch.device, its name or its number; without a number, or for None, the current one)."""
    index = device if device is None or isinstance(device, int) else torch.device(device).index
    return _raw(torch.cuda.current_device() if index is None else index)
