"""Small helpers shared by the host-side modules: dtype codes, stream and pointer access."""
from __future__ import annotations

import contextlib

import torch

from . import _lib

_DTYPE = {torch.float32: _lib.COME_F32, torch.float16: _lib.COME_F16, torch.bfloat16: _lib.COME_BF16}


def dtype_code(dtype: torch.dtype, what: str = "tensor") -> int:
    try:
        return _DTYPE[dtype]
    except KeyError:
        raise RuntimeError(f"{what}: unsupported dtype {dtype}; expected float32, float16 or bfloat16") from None


def require_cuda(t: torch.Tensor, name: str) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{name} must be on CUDA")


def ptr(t):
    return None if t is None else t.data_ptr()


def stream_ptr(device) -> int:
    """Handle of the device's current stream (the bare handle: building a ``torch.cuda.Stream`` on every launch costs more
    than the rest of a small launch's arguments)."""
    index = device.index
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if index is None else index)


_SAME_DEVICE = contextlib.nullcontext()


def on_device(device):
    """Context in which ``device`` is the current CUDA device; nothing to enter or leave when it already is."""
    if device.index is None or device.index == torch.cuda.current_device():
        return _SAME_DEVICE
    return torch.cuda.device(device)
