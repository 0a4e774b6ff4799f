"""Device-memory plumbing for the host layer.

PyTorch is used here for exactly three things: owning device buffers, naming the
current CUDA stream, and (in ``cp``) ``torch.distributed``. No torch operator
runs on the data path; all arithmetic happens inside libb200tri.
"""

from __future__ import annotations

import threading
import weakref
from typing import Any, Mapping

import numpy as np
import torch

# Scratch buffers one thread keeps per device: those of the streams it used last.
STREAMS_KEPT = 4


class _Scratch:
    """One thread's scratch buffers, (device, stream) -> {tag: buffer}, the stream used last at the end."""

    def __init__(self) -> None:
        self.streams: dict[tuple[int, int], dict[str, torch.Tensor]] = {}


_local = threading.local()
_scratches: "weakref.WeakSet[_Scratch]" = weakref.WeakSet()

_cuda_seen = False


def require_cuda() -> None:
    global _cuda_seen
    if _cuda_seen:  # asking the driver again costs a small call microseconds
        return
    if not torch.cuda.is_available():
        raise RuntimeError("foldjax_b200 needs a CUDA device (B200, sm_100a); there is no CPU fallback")
    torch.cuda.init()
    _cuda_seen = True


def stream_ptr() -> int:
    """The current stream of the current device as a raw handle (no Stream object is built)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def place() -> tuple[int, int]:
    """The current device and its current stream as a raw handle."""
    device = torch._C._cuda_getDevice()
    return device, torch._C._cuda_getCurrentRawStream(device)


def workspace(nbytes: int, tag: str = "default", at: tuple[int, int] | None = None) -> torch.Tensor:
    """A grow-only scratch buffer, 1 KiB aligned, of the calling thread, the current device, its
    current stream and ``tag`` (``at``: what ``place()`` gave a caller that has asked).

    Whatever uses a buffer next comes after its previous use in the order of one stream: two streams
    have buffers of their own, and so have two threads, whose launches on one stream may alternate.
    That also makes dropping a buffer safe (it grew, its stream has not been used for a while, its
    thread ended), because the allocator gives its memory to nobody but that stream until then.

    A call that is being captured gets a buffer of the graph's memory pool and none is kept: the graph
    holds the address for as long as it lives, whatever becomes of the buffers kept here, and may be
    replayed beside other calls on its stream."""
    initialized = at is not None or torch.cuda.is_initialized()
    if at is None:
        at = (torch.cuda.current_device(), stream_ptr() if initialized else 0)
    if initialized and torch.cuda.is_current_stream_capturing():
        return torch.empty(int(nbytes) + 1024, dtype=torch.uint8, device=f"cuda:{at[0]}")
    scratch = getattr(_local, "scratch", None)
    if scratch is None:
        scratch = _local.scratch = _Scratch()
        _scratches.add(scratch)
    streams = scratch.streams
    bufs = streams.get(at)
    if bufs is None:
        kept = [k for k in streams if k[0] == at[0]]
        for old in kept[:max(0, len(kept) - STREAMS_KEPT + 1)]:
            streams.pop(old, None)
        bufs = streams[at] = {}
    elif len(streams) > 1:
        streams[at] = streams.pop(at, bufs)  # to the end
    buf = bufs.get(tag)
    if buf is None or buf.numel() < nbytes + 1024:  # callers round the pointer up by up to 1023 B
        bufs.pop(tag, None)
        buf = torch.empty(int(nbytes) + 1024, dtype=torch.uint8, device=f"cuda:{at[0]}")
        bufs[tag] = buf
    return buf


# Batch items share a launch as far as this much scratch memory carries them.
BATCH_WORKSPACE = 2 << 30


def batch_bytes(one: int, batch: int) -> int:
    """Workspace of a batched call: ``one`` item's bytes times the items that run together."""
    return one * max(1, min(batch, BATCH_WORKSPACE // max(one, 1)))


def aligned_ptr(buf: torch.Tensor, align: int = 1024) -> int:
    p = buf.data_ptr()
    return (p + align - 1) // align * align


def check_out(out: torch.Tensor, like: torch.Tensor, name: str = "out") -> torch.Tensor:
    """The caller's result buffer goes to the kernels as a raw pointer, so it must be
    exactly what they write: a contiguous CUDA bf16 tensor of the input's shape on the
    input's device. Anything else would be a write past the buffer, not a Python error."""
    if not isinstance(out, torch.Tensor):
        raise ValueError(f"{name} must be a torch tensor, got {type(out).__name__}")
    if out.dtype != like.dtype:
        raise ValueError(f"{name} must be {like.dtype}, got {out.dtype}")
    if out.shape != like.shape:
        raise ValueError(f"{name} shape {tuple(out.shape)} does not match the input {tuple(like.shape)}")
    if not out.is_contiguous():
        raise ValueError(f"{name} must be contiguous")
    if not out.is_cuda or out.device != like.device:
        raise ValueError(f"{name} must be a CUDA tensor on the input's device ({like.device}), got {out.device}")
    return out


def check_same_shape(t: torch.Tensor, like: torch.Tensor, name: str) -> torch.Tensor:
    if t.shape != like.shape:
        raise ValueError(f"{name} shape {tuple(t.shape)} does not match the input {tuple(like.shape)}")
    return t


def check_device_status() -> None:
    """Read (and clear) the device status word at a point where the host synchronises
    anyway; raises if a kernel gave up on a bounded wait since the last check."""
    from . import _lib

    _lib.device_status()


def release_workspaces() -> None:
    """Drop the scratch buffers of all threads (a call under way keeps its own until it is enqueued)."""
    for scratch in list(_scratches):
        scratch.streams.clear()


def ready(x: Any, dtype: torch.dtype | None) -> bool:
    """Whether the kernels can read ``x`` as it is: a contiguous tensor of ``dtype`` on the current
    device. Most calls bring nothing else, and a ``.to()`` that copies nothing is not free."""
    return (isinstance(x, torch.Tensor) and x.is_cuda and (dtype is None or x.dtype is dtype) and x.is_contiguous()
            and x.get_device() == torch._C._cuda_getDevice())


def to_device(x: Any, dtype: torch.dtype | None = None, device: torch.device | None = None) -> torch.Tensor:
    """numpy / torch (any device) -> contiguous CUDA tensor of `dtype`."""
    if device is None and ready(x, dtype):
        return x
    device = device or torch.device("cuda", torch.cuda.current_device())
    if isinstance(x, np.ndarray):
        if x.dtype.name == "bfloat16":  # ml_dtypes
            t = torch.from_numpy(x.view(np.uint16).copy()).view(torch.bfloat16)
        else:
            t = torch.from_numpy(np.ascontiguousarray(x))
    elif isinstance(x, torch.Tensor):
        t = x
    else:
        t = torch.as_tensor(np.asarray(x))
    t = t.to(device=device, dtype=dtype or t.dtype, non_blocking=True)
    return t.contiguous()


def params_to_device(params: Mapping, dtype: torch.dtype = torch.bfloat16, device=None):
    """Move a nested parameter mapping to the device in the trunk dtype."""
    if isinstance(params, Mapping):
        return {k: params_to_device(v, dtype, device) for k, v in params.items()}
    return to_device(params, dtype, device)


def is_host_array(x: Any) -> bool:
    return isinstance(x, np.ndarray) or (isinstance(x, torch.Tensor) and not x.is_cuda)
