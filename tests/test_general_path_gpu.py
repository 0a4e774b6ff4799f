"""The general-shape path at the edges of its tiles: rows around 64 and 128, one token, channel
counts that leave partial 64-column tiles, every head width class of the split attention core,
batches that do not fit one pass, and operands TMA or 16-byte accesses cannot take.

float32 tolerance: 1e-4 of the output's scale, the bar of the float32 trunk (test_fp32_mode_gpu.py).
bf16: the benchmark's budget (conftest.assert_parity)."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _close_f32(ref, got, where=None):
    scale = max(1.0, float(np.abs(ref).max()))
    err = np.abs(np.asarray(got, np.float64) - ref)
    err = err[where] if where is not None else err
    assert err.max() <= 1e-4 * scale, (err.max(), scale)


@pytest.mark.parametrize("n,c_z,c_hidden", [(1, 64, 64), (63, 72, 40), (65, 128, 136), (129, 256, 128), (40, 512, 8)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_multiplication_edges(cuda_device, n, c_z, c_hidden, dtype):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle import triangle_multiplication_forward

    rng = np.random.default_rng(n + c_z)
    params = orc.random_trimul_params(rng, c_z=c_z, c_hidden=c_hidden, std=0.05, ln_noise=0.1)
    x = rng.standard_normal((1, n, n, c_z)).astype(np.float32)
    mask = (rng.random((1, n, n)) > 0.1).astype(np.float32)
    if dtype == "bfloat16":
        params, x = orc.round_params(params, dtype), orc.round_bf16(x)
    for direction in ("outgoing", "incoming"):
        got = triangle_multiplication_forward(params, x, mask, direction, dtype=dtype, residual=x)
        _lib.device_status()
        update = triangle_multiplication_forward(params, x, mask, direction, dtype=dtype)
        if dtype == "float32":
            ref = orc.triangle_multiplication(params, x, mask, direction, dtype="float64")
            _close_f32(ref, update)
            np.testing.assert_allclose(got, x + update, rtol=0, atol=1e-6)
        else:
            emu = orc.triangle_multiplication(params, x, mask, direction, dtype="bfloat16")
            assert_parity(emu, update, label=f"general trimul n={n} {c_z}/{c_hidden} {direction}")
            assert np.array_equal(got, orc.round_bf16(x + update))


@pytest.mark.parametrize("n,c_z,heads,head_dim", [(1, 64, 4, 16), (64, 72, 3, 24), (65, 64, 2, 64), (129, 40, 5, 8),
                                                  (130, 128, 4, 48)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_edges(cuda_device, n, c_z, heads, head_dim, dtype):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n + c_z)
    params = orc.random_triatt_params(rng, c_z=c_z, heads=heads, c_hidden=head_dim, std=0.1, ln_noise=0.1)
    x = rng.standard_normal((1, n, n, c_z)).astype(np.float32)
    mask = orc.pad_mask(n, 5 if n > 5 else 0)
    if dtype == "bfloat16":
        params, x = orc.round_params(params, dtype), orc.round_bf16(x)
    for starting in (True, False):
        got = triangle_attention_forward(params, x, mask, starting=starting, dtype=dtype)
        _lib.device_status()
        has_key = mask.any(axis=2) if starting else mask.any(axis=1)
        valid = np.broadcast_to(has_key[:, :, None, None] if starting else has_key[:, None, :, None], x.shape)
        if dtype == "float32":
            _close_f32(orc.triangle_attention(params, x, mask, starting=starting, dtype="float64"), got, valid)
        else:
            emu = orc.triangle_attention(params, x, mask, starting=starting, dtype="bfloat16")
            assert_parity(emu, got, where=valid, label=f"general triatt n={n} {c_z} {heads}x{head_dim} starting={starting}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_batches_in_one_and_in_several_passes(cuda_device, monkeypatch, dtype):
    """Five items at once, and two per pass: the same bits as one call per item."""
    from foldjax_b200 import _device as dev
    from foldjax_b200.triangle import triangle_multiplication_forward
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(3)
    n, c_z = 50, 64
    pm = dev.params_to_device(orc.random_trimul_params(rng, c_z=c_z, c_hidden=96, std=0.1), dtype)
    pa = dev.params_to_device(orc.random_triatt_params(rng, c_z=c_z, heads=4, c_hidden=16, std=0.1), dtype)
    x = torch.randn(5, n, n, c_z, device="cuda").to(dtype)
    mask = (torch.rand(5, n, n, device="cuda") > 0.1).float()
    ops = (lambda z, m: triangle_multiplication_forward(pm, z, m, "incoming", residual=z),
           lambda z, m: triangle_attention_forward(pa, z, m, starting=False, residual=z))
    for op in ops:
        single = torch.stack([op(x[b], mask[b]) for b in range(5)])
        assert torch.equal(op(x, mask), single)
        monkeypatch.setattr(dev, "batch_bytes", lambda one, batch: 2 * one)
        assert torch.equal(op(x, mask), single)
        monkeypatch.undo()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_operands_off_the_alignment_grid(cuda_device, dtype):
    from foldjax_b200 import _device as dev
    from foldjax_b200.triangle import triangle_multiplication_forward
    from foldjax_b200.triangle_attention import triangle_attention_forward

    def shifted(node):
        if isinstance(node, dict):
            return {k: shifted(v) for k, v in node.items()}
        buf = torch.empty(node.numel() + 1, dtype=node.dtype, device=node.device)
        buf[1:] = node.reshape(-1)
        return buf[1:].view(node.shape)

    rng = np.random.default_rng(4)
    n, c_z = 37, 64
    pm = dev.params_to_device(orc.random_trimul_params(rng, c_z=c_z, c_hidden=128, std=0.1), dtype)
    pa = dev.params_to_device(orc.random_triatt_params(rng, c_z=c_z, heads=4, c_hidden=16, std=0.1), dtype)
    x = torch.randn(n, n, c_z, device="cuda").to(dtype)
    xs, out = shifted(x), shifted(torch.zeros_like(x))
    assert torch.equal(triangle_multiplication_forward(pm, x, None, "outgoing", residual=x),
                       triangle_multiplication_forward(shifted(pm), xs, None, "outgoing", residual=xs, out=out))
    assert torch.equal(triangle_attention_forward(pa, x, residual=x),
                       triangle_attention_forward(shifted(pa), xs, residual=xs, out=out))
