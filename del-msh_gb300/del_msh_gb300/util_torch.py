"""Helpers shared by the torch front-ends (the checks of
del_msh_dlpack/util_torch.py: shape, dtype and device assertions)."""
from __future__ import annotations

import torch


def assert_shape_dtype_device(t: torch.Tensor, shape, dtype, device):
    assert t.shape == tuple(shape), f"shape {tuple(t.shape)} != {tuple(shape)}"
    assert t.dtype == dtype, f"dtype {t.dtype} != {dtype}"
    assert t.device == device, f"device {t.device} != {device}"


def require_cuda(device: torch.device):
    if device.type != "cuda":
        raise NotImplementedError("del_msh_gb300 runs on CUDA devices only (no CPU path)")


def stream_ptr(device: torch.device) -> int:
    """The current stream of a CUDA device, which becomes the current device."""
    index = device.index
    if torch.cuda.current_device() != index:
        torch.cuda.set_device(device)
        index = torch.cuda.current_device()
    return torch._C._cuda_getCurrentRawStream(index)


def ptr(t):
    """Device address of a contiguous tensor (None -> NULL)."""
    if t is None:
        return None
    assert t.is_contiguous(), "tensor must be contiguous"
    return t.data_ptr()


def plain(t):
    """The tensor itself when it is contiguous, else a contiguous copy outside
    autograd.  The caller keeps it until the launch: its address alone does not
    hold the copy."""
    return t if t is None or t.is_contiguous() else t.detach().contiguous()


def scratch(device: torch.device, nbytes: int) -> torch.Tensor:
    """Working memory for one C-ABI call, from torch's caching allocator (so
    repeated calls reuse it instead of allocating on the device each time);
    its blocks are 512-byte aligned, as the C ABI requires 256."""
    return torch.empty((max(int(nbytes), 1),), dtype=torch.uint8, device=device)
