"""Calls into the library on a device's current stream, with as little Python around them as possible:
a deep stage of the network is a few microseconds of kernels per call, the same as entering
``torch.cuda.device`` and building a ``torch.cuda.Stream`` object."""
import torch

_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_current = getattr(torch._C, "_cuda_getDevice", None)


def call(dev: torch.device, fn, *args) -> int:
    """fn(*args, stream) with ``dev`` current and ``stream`` its current stream."""
    index = dev.index
    if _raw_stream is not None and _current is not None and _current() == index:
        return fn(*args, _raw_stream(index))
    with torch.cuda.device(dev):
        return fn(*args, torch.cuda.current_stream().cuda_stream)
