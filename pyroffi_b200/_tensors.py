"""Tensor plumbing for the ctypes calls: dtype/contiguity coercion, pointers
and the current CUDA stream."""

from __future__ import annotations

import torch


def f32(t) -> torch.Tensor:
    if not isinstance(t, torch.Tensor):
        t = torch.as_tensor(t)
    if t.dtype != torch.float32 or not t.is_contiguous():
        t = t.to(torch.float32).contiguous()
    return t


def i32(t) -> torch.Tensor:
    if not isinstance(t, torch.Tensor):
        t = torch.as_tensor(t)
    if t.dtype != torch.int32 or not t.is_contiguous():
        t = t.to(torch.int32).contiguous()
    return t


def on_device(t: torch.Tensor, device: torch.device) -> torch.Tensor:
    if t.device != device:
        t = t.to(device)
    return t


def ptr(t: torch.Tensor | None) -> int | None:
    # data_ptr() is 0 for a tensor without elements
    return None if t is None else (t.data_ptr() or None)


# The raw handle of the current stream, without the Stream object around it
# (1 us less per call) where torch offers it.
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def stream_ptr(device: torch.device) -> int:
    if _raw_stream is None or type(device) is not torch.device or device.type != "cuda":
        return torch.cuda.current_stream(device).cuda_stream  # raises for a device without streams
    index = device.index
    return _raw_stream(torch.cuda.current_device() if index is None else index)


def require_cuda(*ts: torch.Tensor) -> torch.device:
    dev = None
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda:
            raise ValueError("pyroffi_b200 operators take CUDA tensors (there is no CPU path)")
        dev = t.device if dev is None else dev
        if t.device != dev:
            raise ValueError("all tensors must be on the same CUDA device")
    if dev is None:
        raise ValueError("no tensor given")
    return dev
