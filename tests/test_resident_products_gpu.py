"""Products of the general path with one operand kept in shared memory: runs of several tiles that
end in partial ones, several runs per block (the kept operand refilled, across batch items too), one
and the most k steps that are kept; and two shapes on the other side of the rule, which stream both
operands: one more k step than that, and a single tile to keep the operand for (64 -> 64).

float32: 1e-4 of the output's scale, the float32 trunk's bar; sums of at most 576 products of order
one stay below 576 * 2^-24 of it. bf16: the benchmark's budget (conftest.assert_parity)."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n,c_z,c_hidden", [(1, 20, 128, 264), (1, 150, 64, 64), (1, 12, 512, 128), (1, 12, 576, 128),
                                                  (1, 150, 64, 128), (2, 130, 64, 128)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_gated_projection(cuda_device, batch, n, c_z, c_hidden, dtype):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle import triangle_multiplication_forward

    rng = np.random.default_rng(n + c_z)
    params = orc.round_params(orc.random_trimul_params(rng, c_z=c_z, c_hidden=c_hidden, std=0.05, ln_noise=0.1), dtype)
    x = rng.standard_normal((batch, n, n, c_z)).astype(np.float32)
    x = orc.round_bf16(x) if dtype == "bfloat16" else x
    mask = (rng.random((batch, n, n)) > 0.1).astype(np.float32)
    got = triangle_multiplication_forward(params, x, mask, "outgoing", dtype=dtype)
    _lib.device_status()
    if dtype == "float32":
        ref = orc.triangle_multiplication(params, x, mask, "outgoing", dtype="float64")
        assert np.abs(got - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    else:
        assert_parity(orc.triangle_multiplication(params, x, mask, "outgoing", dtype=dtype), got, label=f"{batch} x {n} {c_z}/{c_hidden}")


@pytest.mark.parametrize("batch,n,c_z,heads,head_dim", [(1, 150, 64, 4, 16), (1, 40, 128, 12, 32), (1, 30, 136, 12, 32),
                                                        (2, 130, 64, 4, 16)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_projection(cuda_device, batch, n, c_z, heads, head_dim, dtype):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n + c_z)
    params = orc.round_params(orc.random_triatt_params(rng, c_z=c_z, heads=heads, c_hidden=head_dim, std=0.05, ln_noise=0.1), dtype)
    x = rng.standard_normal((batch, n, n, c_z)).astype(np.float32)
    x = orc.round_bf16(x) if dtype == "bfloat16" else x
    mask = np.ones((batch, n, n), np.float32)
    got = triangle_attention_forward(params, x, mask, dtype=dtype)
    _lib.device_status()
    if dtype == "float32":
        ref = orc.triangle_attention(params, x, mask, True, dtype="float64")
        assert np.abs(got - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    else:
        assert_parity(orc.triangle_attention(params, x, mask, True, dtype=dtype), got, label=f"{batch} x {n} {c_z} {heads}x{head_dim}")
