"""Tensor plumbing for the ctypes calls: device placement, dtype and layout
checks, raw pointers and the current CUDA stream."""
import math

import numpy as np
import torch


_devices = {}  # index -> torch.device, filled once CUDA has been seen


def device():
    """The current CUDA device. (Each query of torch.cuda.is_available() and a
    new torch.device cost about as much as the allocation they precede: an
    empty() took 3.3 us of host time, 1.6 of them torch's.)"""
    if not _devices and not torch.cuda.is_available():
        raise RuntimeError("libnerfgb needs a CUDA device (sm_103); none is visible")
    i = torch.cuda.current_device()
    d = _devices.get(i)
    if d is None:
        d = _devices[i] = torch.device("cuda", i)
    return d


def as_cuda(x, dtype=torch.float32, shape=None, name="tensor"):
    """Returns x as a contiguous CUDA tensor of `dtype` (copying only when x is
    on the host, has another dtype or is strided)."""
    if not (isinstance(x, torch.Tensor) and x.is_cuda and x.dtype == dtype and x.is_contiguous()):
        if isinstance(x, np.ndarray):
            x = torch.from_numpy(np.ascontiguousarray(x))
        if not isinstance(x, torch.Tensor):
            x = torch.as_tensor(x)
        if x.device.type != "cuda":
            x = x.to(device())
        if x.dtype != dtype:
            x = x.to(dtype)
        if not x.is_contiguous():
            x = x.contiguous()
    if shape is not None and x.shape != shape:
        want = tuple(shape)
        if tuple(x.shape) != want:
            if x.numel() == math.prod(want):
                x = x.reshape(want)
            else:
                raise ValueError(f"{name}: expected shape {want}, got {tuple(x.shape)}")
    return x


def ptr(x):
    return None if x is None else x.data_ptr()


def stream():
    # the raw handle of torch.cuda.current_stream(), without building the
    # Stream object (3 us)
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def empty(*shape, dtype=torch.float32):
    return torch.empty(*shape, dtype=dtype, device=device())
