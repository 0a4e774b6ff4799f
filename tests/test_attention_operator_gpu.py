"""The attention-core operator on the caller's [B, I, H, token, D] operands: sizes around the
64-key and 128-query tiles, key counts that TMA can and cannot read in place, float32 operands,
batches and slices off the 16-byte grid, against the oracle."""

import numpy as np
import pytest
import torch

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,n_i,n_j,n_k,v_f32,bias_f32,offset", [
    (1, 1, 1, 1, False, False, False), (1, 3, 128, 64, False, False, False), (2, 5, 129, 65, False, False, False),
    (1, 4, 100, 72, True, True, False), (2, 7, 33, 200, False, True, True), (1, 2, 257, 130, True, False, True)])
def test_attention_core_operator(cuda_device, b, n_i, n_j, n_k, v_f32, bias_f32, offset):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import attention_core

    rng = np.random.default_rng(n_j * 1000 + n_k)
    draw = lambda *shape, scale=1.0: orc.round_bf16(rng.normal(size=shape, scale=scale).astype(np.float32))
    q, k, v = draw(b, n_i, 4, n_j, 32, scale=0.5), draw(b, n_i, 4, n_k, 32, scale=0.5), draw(b, n_i, 4, n_k, 32)
    tb = draw(b, 1, 4, n_j, n_k, scale=2.0)
    keep = rng.random((b, n_i, n_k)) > 0.2
    keep[..., 0] = True
    mb = np.where(keep[:, :, None, None, :], np.float32(0), np.float32(-1e9))
    ref = orc.attention_core(q, k, v, tb, mb, dtype="bfloat16")

    def t(a, dtype):
        x = torch.from_numpy(a).to(cuda_device).to(dtype)
        if offset:  # a view whose first element is off the 16-byte grid
            x = torch.cat([x.new_zeros(1), x.reshape(-1)])[1:].view(a.shape)
        return x

    bf, f32 = torch.bfloat16, torch.float32
    got = attention_core(t(q, bf), t(k, bf), t(v, f32 if v_f32 else bf), t(tb, f32 if bias_f32 else bf), t(mb, f32))
    _lib.device_status()
    assert got.shape == ref.shape and got.dtype == (f32 if v_f32 else bf)
    assert_parity(ref, got.float().cpu().numpy(), label=f"operator {b}x{n_i}x{n_j}x{n_k}")


@pytest.mark.parametrize("n_k", [1, 63, 65, 511, 513, 575, 1025])
@pytest.mark.parametrize("bias_f32", [False, True])
def test_copied_bias_rows(cuda_device, n_k, bias_f32):
    """The bias where the preparation copies it: rows that end anywhere in the 512 elements a warp takes at a time, and a
    last block of rows that is not full."""
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import attention_core

    n_j = 9
    rng = np.random.default_rng(n_k)
    draw = lambda *shape, scale=1.0: orc.round_bf16(rng.normal(size=shape, scale=scale).astype(np.float32))
    q, k, v = draw(1, 2, 4, n_j, 32, scale=0.5), draw(1, 2, 4, n_k, 32, scale=0.5), draw(1, 2, 4, n_k, 32)
    tb, mb = draw(1, 1, 4, n_j, n_k, scale=2.0), np.zeros((1, 2, 1, 1, n_k), np.float32)
    ref = orc.attention_core(q, k, v, tb, mb, dtype="bfloat16")
    t = lambda a, dtype=torch.bfloat16: torch.from_numpy(a).to(cuda_device).to(dtype)
    got = attention_core(t(q), t(k), t(v), t(tb, torch.float32 if bias_f32 else torch.bfloat16), t(mb, torch.float32))
    _lib.device_status()
    assert_parity(ref, got.float().cpu().numpy(), label=f"operator, bias rows of {n_k}")
