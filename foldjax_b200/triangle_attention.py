"""Triangle attention (starting / ending node) on B200 - host side.

Mirrors ``triangle_attention_forward`` of the reference
(src/foldjax/models/boltz2/models/triangle/triangle_attention.py:79-162) and the
attention-core operator its fused backends implement
(``pallas_attention_core``, triangle_attention_pallas.py:180; ``cueq_attention_core``,
src/foldjax/models/_cueq.py:66). Same argument names and meaning; chunking knobs
are accepted and ignored, as the reference's fused backends do.
"""

from __future__ import annotations

import ctypes as C
import math
from functools import lru_cache
from typing import Any, Mapping

import numpy as np
import torch

from . import _device as dev
from . import _lib
from .triangle import C_Z, _as_leaves, _check_leaves, _check_pair, _pair_mask, _ptr, _unfold, resolve_dtype

HEADS = 4
HEAD_DIM = 32
FLOAT_MAX = 3.4028234e38

_FIELDS = ("norm_scale", "norm_bias", "w_bias", "w_q", "w_k", "w_v", "w_g", "w_o")


@lru_cache(maxsize=64)
def _shapes(c_z: int, heads: int, width: int) -> list[tuple]:
    return [(c_z,), (c_z,), (c_z, heads), (c_z, width), (c_z, width), (c_z, width), (c_z, width), (width, c_z)]


def triangle_attention_forward(
    params: Mapping[str, Any],
    x: Any,
    mask: Any | None = None,
    starting: bool = True,
    inf: float = 1e9,
    eps: float = 1e-5,
    chunk_size: int = 128,
    q_chunk_size: int | None = None,
    matmul_precision: str = "highest",
    triangle_backend: str = "b200",
    *,
    residual: Any | None = None,
    out: torch.Tensor | None = None,
    dtype: str | None = None,
):
    """Boltz TriangleAttention, starting or ending node.

    ``x`` is ``[B, N, N, 128]`` (or ``[N, N, 128]``), ``mask`` ``[B, N, N]`` or None (= ones).
    ``dtype`` selects the trunk: "bfloat16" (default) or "float32" (float32 accuracy
    throughout, the reference's float32 trunk, 1e-4); a float32 CUDA tensor selects
    float32 by itself. ``params`` is the reference's mapping ``{"layer_norm": {scale,
    bias}, "linear": {kernel [128, 4]}, "mha": {"linear_q" | "linear_k" |
    "linear_v" | "linear_g" | "linear_o": {kernel [128, 128]}}}``. Device tensors in
    -> device tensor out; NumPy / CPU tensors in -> copied to the GPU and back.
    """
    if triangle_backend != "b200":
        raise ValueError(f"Unsupported triangle_backend: {triangle_backend!r}")
    if matmul_precision.lower() not in ("highest", "float32", "fp32", "default", "tensorfloat32", "tf32"):
        raise ValueError(f"Unsupported matmul_precision: {matmul_precision!r}")
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
    norm, mha = params["layer_norm"], params["mha"]
    leaves = _as_leaves([norm["scale"], norm["bias"], params["linear"]["kernel"], mha["linear_q"]["kernel"], mha["linear_k"]["kernel"],
                         mha["linear_v"]["kernel"], mha["linear_g"]["kernel"], mha["linear_o"]["kernel"]], tdt)
    heads = leaves[2].shape[-1]
    width = leaves[6].shape[-1]
    head_dim = width // max(heads, 1)
    want = _shapes(c_z, heads, width)
    if [t.shape for t in leaves] != want:
        _check_leaves(dict(zip(_FIELDS, leaves)), dict(zip(_FIELDS, want)), "triangle attention",
                      f"c_z = {c_z}, {heads} heads x {head_dim}")
    if heads * head_dim != width or head_dim not in (8, 16, 24, 32, 48, 64):
        raise ValueError(f"libb200tri takes head widths 8, 16, 24, 32, 48 and 64; got {heads} heads over {width} channels")
    nbytes = _lib.workspace_bytes("b200tri_triatt_workspace_bytes_shape", n, code, c_z, heads, head_dim)
    if b > 1 and (code, c_z, heads, head_dim) != (_lib.DTYPE_BF16, C_Z, HEADS, HEAD_DIM):
        nbytes = dev.batch_bytes(nbytes, b)  # the general path takes several items per launch
    at = dev.place()
    ws = dev.workspace(nbytes, "triatt", at)
    if not -FLOAT_MAX < inf < FLOAT_MAX:
        inf = C.c_float(inf).value
    args = _lib.pack_triatt(n, int(bool(starting)), heads, head_dim, inf, float(eps), xd.data_ptr(), _ptr(md),
                            *[v.data_ptr() for v in leaves], _ptr(rd), out.data_ptr(), dev.aligned_ptr(ws),
                            nbytes, code, c_z, b)
    if b:  # (an empty batch has an empty result)
        _lib.check(lib.b200tri_triatt_forward_packed(args, at[1]))
    result = _unfold(out, lead)
    if host_in:
        host = result.float().cpu() if numpy_in else result.cpu()
        dev.check_device_status()  # the copy synchronised: a kernel that gave up on a wait shows here
        return host.numpy() if numpy_in else host
    return result


def attention_core(q, k, v, tri_bias, mask_bias, scale: float | None = None):
    """The attention-core operator: ``core(q, k, v, tri_bias, mask_bias[, scale]) -> out``.

    q/k/v ``[B, I, H, J, D]`` device tensors (q pre-scaled unless ``scale`` is given, the
    cuEquivariance convention of src/foldjax/models/_cueq.py:66-121: q is then multiplied by
    ``scale`` cast to q's dtype and the product rounded to that dtype, as the reference's
    Protenix path does, triangle.py:563,792), ``tri_bias [B, 1, H, J, K]``, ``mask_bias
    [B, I, 1, 1, K]`` additive fp32 (0, a soft bias, -1e9 or -inf). Returns ``[B, I, H, J, D]``
    in ``v.dtype``. Leading axes beyond five are folded into B.

    The additive mask bias goes to the kernel as it is (no round trip through a 0/1 mask), so
    soft and hard entries can be mixed; a row with no kept key comes out as the uniform average
    over its keys, the convention of the finite -1e9 mask (triangle_attention.py:138-142), not as
    the zeros of the reference's 2-D ring (src/foldjax/models/_cp_attention.py:380-385). A dropped key
    (mask bias of -30000 or less) scores -30000 and so has no weight beside kept keys that score above
    some -29980; a query whose kept keys all score less (a pair bias used as a mask) gives its dropped keys weight.
    Enqueue-only: nothing here waits for the device. bf16 operands are read where they are (the
    library transposes v, builds the mask rows and, only where its rows are off TMA's 16-byte
    grid or float32, copies the bias); other element types are converted first.
    """
    dev.require_cuda()
    lib = _lib.load()
    lead = q.shape[:-4]
    bsz = math.prod(lead)
    n_i, h, n_j, d = q.shape[-4:]
    n_k = k.shape[-2]
    if (h, d) != (HEADS, HEAD_DIM):
        raise ValueError(f"libb200tri is built for 4 heads x 32; got {h} x {d}")
    if mask_bias.shape[-4:] != (n_i, 1, 1, n_k) or tri_bias.shape[-4:] != (1, h, n_j, n_k):
        raise ValueError(f"mask_bias {tuple(mask_bias.shape)} / tri_bias {tuple(tri_bias.shape)} do not match "
                         f"q {tuple(q.shape)} and k {tuple(k.shape)}")
    for name, t, count in (("k", k, bsz * n_i * h * n_k * d), ("v", v, bsz * n_i * h * n_k * d),
                           ("tri_bias", tri_bias, bsz * h * n_j * n_k), ("mask_bias", mask_bias, bsz * n_i * n_k)):
        if t.numel() != count:
            raise ValueError(f"{name} shape {tuple(t.shape)} does not match q {tuple(q.shape)}")
    qd = _operand(q, torch.bfloat16)
    if scale is not None:
        # one bf16 rounding of q times the bf16 value of scale
        qd = qd * torch.tensor(float(scale), dtype=torch.bfloat16).item()
    kd = _operand(k, torch.bfloat16)
    vd = _operand(v, v.dtype if v.dtype in (torch.bfloat16, torch.float32) else torch.float32)
    bd = _operand(tri_bias, tri_bias.dtype if tri_bias.dtype in (torch.bfloat16, torch.float32) else torch.bfloat16)
    md = _operand(mask_bias, torch.float32)
    out = torch.empty(q.shape, dtype=torch.bfloat16, device=q.device)
    nbytes = _lib.workspace_bytes("b200tri_attention_core_workspace_bytes", n_i, n_j, n_k)
    at = dev.place()
    ws = dev.workspace(nbytes, "attention_core", at)
    args = _lib.pack_attention_core(bsz, n_i, n_j, n_k, h, d, int(vd.dtype is torch.float32), int(bd.dtype is torch.float32),
                                    qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), bd.data_ptr(), md.data_ptr(),
                                    out.data_ptr(), dev.aligned_ptr(ws), nbytes)
    if bsz:  # (an empty batch has an empty result)
        _lib.check(lib.b200tri_attention_core_packed(args, at[1]))
    return out if v.dtype is torch.bfloat16 else out.to(v.dtype)


def _operand(t: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """``t`` as the library reads it: dense, of ``dtype`` and 16-byte aligned (a slice need not be)."""
    if t.dtype is not dtype or not t.is_contiguous():
        t = t.to(dtype).contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()
