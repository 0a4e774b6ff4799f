"""Triangle multiplicative update on B200 - host side.

Mirrors ``triangle_multiplication_forward`` of the reference
(src/foldjax/models/boltz2/models/triangle/triangle.py:33-129): same argument
names and meaning, same parameter mapping, same error text for a bad direction.
The arithmetic runs in libb200tri (hand-written sm_100a kernels); nothing here
falls back to another implementation.
"""

from __future__ import annotations

from functools import lru_cache
from typing import Any, Mapping

import numpy as np
import torch

from . import _device as dev
from . import _lib

C_Z = 128  # channel width of the tensor-core specialisation (other widths run the general path)


def _ptr(t: torch.Tensor | None) -> int:
    return 0 if t is None else t.data_ptr()


def _check_pair(x: torch.Tensor) -> tuple[torch.Tensor, Any]:
    """-> (the pair tensor as [B, N, N, C], the caller's leading shape). A missing batch axis is
    added and leading axes beyond one are folded into B, the way the reference's fused
    wrappers do it (src/foldjax/models/_cueq.py:89-121); the second item is what to restore."""
    shape = tuple(x.shape)
    if len(shape) < 3 or shape[-2] != shape[-3]:
        raise ValueError(f"expected a pair tensor [B, N, N, C], got shape {shape}")
    if shape[-1] % 8 or shape[-1] > 1024:
        raise ValueError(f"libb200tri takes channel counts that are multiples of 8 up to 1024; got {shape[-1]} channels")
    return x if len(shape) == 4 else x.reshape((-1,) + shape[-3:]), shape[:-3]


def _unfold(t: torch.Tensor, lead: tuple) -> torch.Tensor:
    return t if len(lead) == 1 else t.reshape(tuple(lead) + tuple(t.shape[1:]))


def _as_leaf(node: Any, dtype: torch.dtype) -> torch.Tensor:
    if not isinstance(node, torch.Tensor) or node.dtype is not dtype or not node.is_cuda:
        node = dev.to_device(node, dtype)
    return node if node.is_contiguous() else node.contiguous()


def _leaf(params: Mapping, *path: str, dtype: torch.dtype = torch.bfloat16) -> torch.Tensor:
    node: Any = params
    for key in path:
        node = node[key]
    return _as_leaf(node, dtype)


def _as_leaves(nodes: list, dtype: torch.dtype) -> list[torch.Tensor]:
    """``_as_leaf`` of each; nearly always they are leaves already, and a call for each takes three times as long as
    the checks in line."""
    for node in nodes:
        if not (isinstance(node, torch.Tensor) and node.dtype is dtype and node.is_cuda and node.is_contiguous()):
            return [_as_leaf(node, dtype) for node in nodes]
    return nodes


def _check_leaves(leaves: Mapping[str, torch.Tensor], want: Mapping[str, tuple], what: str, where: str) -> None:
    for name, shape in want.items():
        if leaves[name].shape != shape:
            raise ValueError(f"{what} parameter {name} has shape {tuple(leaves[name].shape)}, expected {shape} for {where}")


def _pair_mask(mask: Any, b: int, n: int, x: Any) -> torch.Tensor | None:
    """The pair mask of a call as float32 with b * n * n values (None = ones)."""
    if mask is None:
        return None
    md = dev.to_device(mask, torch.float32)
    shape = md.shape
    if shape != (b, n, n) and (len(shape) < 2 or shape[-2:] != (n, n) or md.numel() != b * n * n):
        raise ValueError(f"mask shape {tuple(shape)} does not match pair tensor {tuple(x.shape)}")
    return md


def resolve_dtype(x: Any, dtype: str | None) -> tuple[torch.dtype, int]:
    """Trunk dtype of a call: ``dtype`` if given ("bfloat16" / "float32"), else float32 for a
    float32 CUDA tensor and bfloat16 for everything else (host arrays are float32 containers
    of either trunk, so they say nothing). Returns (torch dtype, the C ABI's dtype code)."""
    if dtype is None:
        if isinstance(x, torch.Tensor) and x.is_cuda and x.dtype is torch.float32:
            return torch.float32, _lib.DTYPE_F32
        return torch.bfloat16, _lib.DTYPE_BF16
    name = {"bf16": "bfloat16", "fp32": "float32"}.get(str(dtype), str(dtype))
    if name == "bfloat16":
        return torch.bfloat16, _lib.DTYPE_BF16
    if name == "float32":
        return torch.float32, _lib.DTYPE_F32
    raise ValueError(f"Unsupported dtype: {dtype!r} (expected 'bfloat16' or 'float32')")


_FIELDS = ("norm_in_scale", "norm_in_bias", "p_in", "g_in", "norm_out_scale", "norm_out_bias", "p_out", "g_out")


@lru_cache(maxsize=64)
def _shapes(c_z: int, c_hidden: int) -> list[tuple]:
    return [(c_z,), (c_z,), (c_z, 2 * c_hidden), (c_z, 2 * c_hidden), (c_hidden,), (c_hidden,), (c_hidden, c_z), (c_z, c_z)]


def triangle_multiplication_forward(
    params: Mapping[str, Mapping[str, Any]],
    x: Any,
    mask: Any,
    direction: str,
    eps: float = 1e-5,
    chunk_size: int = 128,
    glu_backend: str = "xla",
    contraction_precision: str = "float32",
    *,
    residual: Any | None = None,
    out: torch.Tensor | None = None,
    dtype: str | None = None,
):
    """Boltz triangle multiplication, outgoing or incoming.

    ``x`` is ``[B, N, N, 128]`` (or ``[N, N, 128]``), ``mask`` is ``[B, N, N]`` or None.
    ``dtype`` selects the trunk: "bfloat16" (default; bf16 storage, fp32 accumulation) or
    "float32" (every step in float32, the contraction as split-bf16 products on the tensor
    cores; the reference's float32 trunk, 1e-4). A float32 CUDA tensor selects float32 by
    itself. Device tensors in -> device tensor out; NumPy / CPU
    tensors in -> the inputs are copied to the GPU, the result is copied back and
    returned as the same kind of array (the end-to-end path).

    ``chunk_size``, ``glu_backend`` and ``contraction_precision`` are accepted for
    signature compatibility: a fused backend has nothing to chunk, and the
    contraction always accumulates in fp32 on the tensor cores (the reference's
    default "float32" mode).  ``residual`` (optional) fuses the caller's
    ``z + update``.
    """
    if direction not in ("outgoing", "incoming"):
        raise ValueError(f"Unsupported triangle multiplication direction: {direction!r}")
    if contraction_precision not in ("float32", "bf16"):
        raise ValueError(f"Unsupported contraction_precision: {contraction_precision!r}")
    dev.require_cuda()
    lib = _lib.load()
    host_in = dev.is_host_array(x)
    numpy_in = isinstance(x, np.ndarray)
    tdt, code = resolve_dtype(x, dtype)
    xd, lead = _check_pair(dev.to_device(x, tdt))
    b, n, _, c_z = xd.shape
    md = _pair_mask(mask, b, n, x)
    rd = None
    if residual is not None:
        rd = xd if residual is x else _check_pair(dev.to_device(residual, tdt))[0]
        dev.check_same_shape(rd, xd, "residual")
    if out is None:
        out = torch.empty_like(xd)
    else:
        if isinstance(out, torch.Tensor) and out.numel() == xd.numel() and out.is_contiguous():
            out = out.view(xd.shape) if tuple(out.shape[-3:]) == tuple(xd.shape[-3:]) else out
        dev.check_out(out, xd)
    norm_in, norm_out = params["norm_in"], params["norm_out"]
    leaves = _as_leaves([norm_in["scale"], norm_in["bias"], params["p_in"]["kernel"], params["g_in"]["kernel"],
                         norm_out["scale"], norm_out["bias"], params["p_out"]["kernel"], params["g_out"]["kernel"]], tdt)
    c_hidden = leaves[6].shape[0]
    want = _shapes(c_z, c_hidden)
    if [t.shape for t in leaves] != want:
        _check_leaves(dict(zip(_FIELDS, leaves)), dict(zip(_FIELDS, want)), "triangle multiplication",
                      f"c_z = {c_z}, c_hidden = {c_hidden}")
    if c_hidden % 8 or c_hidden > 1024:
        raise ValueError(f"libb200tri takes hidden widths that are multiples of 8 up to 1024; got {c_hidden}")
    nbytes = _lib.workspace_bytes("b200tri_trimul_workspace_bytes_shape", n, code, c_z, c_hidden)
    if b > 1 and (code, c_z, c_hidden) != (_lib.DTYPE_BF16, C_Z, C_Z):
        nbytes = dev.batch_bytes(nbytes, b)  # the general path takes several items per launch
    at = dev.place()
    ws = dev.workspace(nbytes, "trimul", at)
    args = _lib.pack_trimul(n, int(direction == "incoming"), float(eps), xd.data_ptr(), _ptr(md),
                            *[v.data_ptr() for v in leaves], _ptr(rd), out.data_ptr(), dev.aligned_ptr(ws),
                            nbytes, code, c_z, c_hidden, b)
    if b:  # (an empty batch has an empty result)
        _lib.check(lib.b200tri_trimul_forward_packed(args, at[1]))
    result = _unfold(out, lead)
    if host_in:
        host = result.float().cpu() if numpy_in else result.cpu()
        dev.check_device_status()  # the copy synchronised: a kernel that gave up on a wait shows here
        return host.numpy() if numpy_in else host
    return result
