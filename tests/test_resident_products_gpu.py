"""Products of the general path with one operand kept in shared memory: runs of several tiles that
end in partial ones, several runs per block, one and the most k steps that are kept, and one more
than that (both operands streamed again).

float32: 1e-4 of the output's scale, the float32 trunk's bar; sums of at most 576 products of order
one stay below 576 * 2^-24 of it. bf16: the benchmark's budget (conftest.assert_parity)."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c_z,c_hidden", [(20, 128, 264), (150, 64, 64), (12, 512, 128), (12, 576, 128)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_gated_projection(cuda_device, n, c_z, c_hidden, dtype):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle import triangle_multiplication_forward

    rng = np.random.default_rng(n + c_z)
    params = orc.round_params(orc.random_trimul_params(rng, c_z=c_z, c_hidden=c_hidden, std=0.05, ln_noise=0.1), dtype)
    x = rng.standard_normal((1, n, n, c_z)).astype(np.float32)
    x = orc.round_bf16(x) if dtype == "bfloat16" else x
    mask = (rng.random((1, n, n)) > 0.1).astype(np.float32)
    got = triangle_multiplication_forward(params, x, mask, "outgoing", dtype=dtype)
    _lib.device_status()
    if dtype == "float32":
        ref = orc.triangle_multiplication(params, x, mask, "outgoing", dtype="float64")
        assert np.abs(got - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    else:
        assert_parity(orc.triangle_multiplication(params, x, mask, "outgoing", dtype=dtype), got, label=f"{n} {c_z}/{c_hidden}")


@pytest.mark.parametrize("n,c_z,heads,head_dim", [(150, 64, 4, 16), (40, 128, 12, 32), (30, 136, 12, 32)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_projection(cuda_device, n, c_z, heads, head_dim, dtype):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n + c_z)
    params = orc.round_params(orc.random_triatt_params(rng, c_z=c_z, heads=heads, c_hidden=head_dim, std=0.05, ln_noise=0.1), dtype)
    x = rng.standard_normal((1, n, n, c_z)).astype(np.float32)
    x = orc.round_bf16(x) if dtype == "bfloat16" else x
    mask = np.ones((1, n, n), np.float32)
    got = triangle_attention_forward(params, x, mask, dtype=dtype)
    _lib.device_status()
    if dtype == "float32":
        ref = orc.triangle_attention(params, x, mask, True, dtype="float64")
        assert np.abs(got - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    else:
        assert_parity(orc.triangle_attention(params, x, mask, True, dtype=dtype), got, label=f"{n} {c_z} {heads}x{head_dim}")
