"""The current CUDA stream as an object, without building one at every call.

``torch.cuda.current_stream()`` builds a ``Stream`` each time, some 6 us of host time, and ``Event.record()`` without a
stream does the same: a decode step of a small model, whose kernels take 65 us, records two events.  The raw handle
of the current stream costs a tenth of a microsecond; the object that goes with it is kept, a few of them per thread."""

from __future__ import annotations

import threading

import torch

_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_raw_device = getattr(torch._C, "_cuda_getDevice", None)
_kept = threading.local()
_MOST = 16


def current_stream():
    """The stream that work of this thread goes to now."""
    if _raw_stream is None or _raw_device is None:
        return torch.cuda.current_stream()
    device = _raw_device()
    key = (device, _raw_stream(device))
    streams = _kept.__dict__.setdefault("streams", {})
    stream = streams.get(key)
    if stream is None:
        if len(streams) >= _MOST:
            streams.clear()
        stream = streams[key] = torch.cuda.current_stream()
    return stream
