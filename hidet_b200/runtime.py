"""Device plumbing for the host layer: dtype codes, pointers, streams and the scratch workspace.

torch is used for device memory and streams only; every computation happens inside
libhidet_b200q.so.
"""
from __future__ import annotations

from typing import Dict, Optional, Tuple

import torch

from . import ffi, native

FLOAT_CODES = {torch.float16: ffi.F16, torch.bfloat16: ffi.BF16, torch.float32: ffi.F32}
QUANT_CODES = {torch.int8: ffi.I8, torch.int16: ffi.I16}
QUANT_NAMES = {'int8': torch.int8, 'i8': torch.int8, 'int16': torch.int16, 'i16': torch.int16}


def require_cuda(t: torch.Tensor, name: str) -> None:
    if not isinstance(t, torch.Tensor):
        raise TypeError('{} must be a torch.Tensor, got {}'.format(name, type(t).__name__))
    if not t.is_cuda:
        raise ffi.BackendException(
            '{} lives on {}: hidet_b200 runs on CUDA devices only and has no CPU implementation'.format(name, t.device)
        )


def current_stream_ptr(device: torch.device) -> int:
    """The stream kernels are launched on: torch's current stream, as in the reference, whose runtime
    asks torch for it through a callback (src/hidet/runtime/cuda/context.cpp:78-88)."""
    return torch.cuda.current_stream(device).cuda_stream


class _Workspaces:
    """Grow-only, zero-initialised scratch per (device, stream), the role request_cuda_workspace
    plays in the reference (src/hidet/runtime/cuda/context.cpp:31-49,90-104).  The library keeps the
    part that must be zero (its tile counters) zero between calls, so a buffer is cleared only when it
    is created."""

    def __init__(self):
        self._buffers: Dict[Tuple[int, int], torch.Tensor] = {}

    def get(self, device: torch.device, nbytes: int) -> Tuple[int, int]:
        if nbytes == 0:
            return 0, 0
        index = device.index if device.index is not None else torch.cuda.current_device()
        key = (index, current_stream_ptr(device))
        buf = self._buffers.get(key)
        if buf is None or buf.numel() < nbytes:
            size = 1 << max(20, (nbytes - 1).bit_length())
            buf = torch.zeros(size, dtype=torch.uint8, device=torch.device('cuda', index))
            self._buffers[key] = buf
        native.set_scratch(*key, buf.data_ptr(), buf.numel())  # for the native host path, which may be younger than the buffer
        return buf.data_ptr(), buf.numel()

    def clear(self) -> None:
        self._buffers.clear()
        native.clear_scratch()

    def swap(self, device: torch.device, stream: int, buffer: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
        """Puts `buffer` (None: nothing, a new one is made when it is needed) in the place of a stream's scratch and
        returns what was there.  A captured graph takes the buffer its launches were recorded with into its own keeping
        this way: streams come from a small pool, so a later graph or eager call may run on the same one, and must neither
        share the buffer nor replace it by a larger one while the graph still writes to it."""
        index = device.index if device.index is not None else torch.cuda.current_device()
        before = self._buffers.pop((index, stream), None)
        if buffer is not None:
            self._buffers[(index, stream)] = buffer
        native.set_scratch(index, stream, buffer.data_ptr() if buffer is not None else 0, buffer.numel() if buffer is not None else 0)
        return before


workspaces = _Workspaces()
