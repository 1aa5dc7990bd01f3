"""Current stream and stream switch for the call paths of the buffers.

``torch.cuda.current_stream()`` and ``torch.cuda.stream(s)`` look the current device up through the availability check
(environment, NVML) on every call, 5-7 us each, and a dispatch + combine pair makes fourteen of these calls.  Both helpers
ask the runtime for the current device instead; what they return and set is the same.
"""
import torch


def current_stream() -> 'torch.cuda.Stream':
    """``torch.cuda.current_stream()`` (CUDA must be initialised: a buffer exists)."""
    return torch.cuda.current_stream(torch._C._cuda_getDevice())


class on_stream:
    """``with torch.cuda.stream(stream)``."""
    __slots__ = ('_stream', '_previous', '_general')

    def __init__(self, stream: 'torch.cuda.Stream'):
        self._stream = stream

    def __enter__(self) -> None:
        # a stream of another device also switches the device: left to PyTorch
        self._general = None
        if self._stream.device_index != torch._C._cuda_getDevice():
            self._general = torch.cuda.stream(self._stream)
            self._general.__enter__()
        else:
            self._previous = current_stream()
            torch.cuda.set_stream(self._stream)

    def __exit__(self, *exc) -> None:
        if self._general is not None:
            self._general.__exit__(*exc)
        else:
            torch.cuda.set_stream(self._previous)
