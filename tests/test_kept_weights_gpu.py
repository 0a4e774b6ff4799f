"""Products of the general bf16 path whose weights stay in shared memory (piece_gemm_resident_kernel, ONCE): one and two
k steps; fewer, as many and more units of rows than SMs, so that the ring of rows goes round; runs of one tile where all of
them fit the SMs at once; column groups of two weights in a tile, a last group that no weight has, as many heads as a group of
columns. And shapes on the other side of the rules: weights that leave no room for two units' rows, three k steps; of
those a little fewer and a little more tiles of rows than make keeping the rows pay; heads of up to 64 columns in all, which
stream in tiles of 64 columns up to one and a quarter tiles of rows an SM (153 tokens; 154 are the first behind it).

Tolerance: the benchmark's bf16 budget (conftest.assert_parity). Its bound of four units in the last place is for sums of many
products: one flipped rounding of a gated value y moves an output by 2^-8 |y w|, here up to 2^-8 * 4 * 0.4, which is 0.07 of the
RMS of a sum of eight such products, so heads of eight columns in all stand on no side of it."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n,c_z,c_hidden", [(1, 5, 64, 128), (1, 74, 64, 128), (1, 75, 64, 128), (3, 100, 64, 128), (1, 131, 40, 72),
                                                  (1, 149, 128, 136), (1, 130, 72, 64), (1, 130, 64, 264), (1, 100, 136, 128)])
def test_gated_projection(cuda_device, batch, n, c_z, c_hidden):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle import triangle_multiplication_forward

    rng = np.random.default_rng(n + c_hidden)
    params = orc.round_params(orc.random_trimul_params(rng, c_z=c_z, c_hidden=c_hidden, std=0.05, ln_noise=0.1), "bfloat16")
    x = orc.round_bf16(rng.standard_normal((batch, n, n, c_z)).astype(np.float32))
    mask = np.ones((batch, n, n), np.float32)
    mask[:, :, n // 2] = 0.0  # (runs of pairs with a mask and without)
    got = triangle_multiplication_forward(params, x, mask, "incoming", dtype="bfloat16")
    _lib.device_status()
    assert_parity(orc.triangle_multiplication(params, x, mask, "incoming", dtype="bfloat16"), got, label=f"{batch} x {n} {c_z}/{c_hidden}")


@pytest.mark.parametrize("batch,n,c_z,heads,head_dim", [(1, 5, 64, 4, 16), (1, 97, 64, 4, 16), (1, 98, 64, 8, 8), (3, 100, 64, 4, 16),
                                                        (1, 131, 40, 2, 24), (1, 137, 72, 2, 48), (1, 90, 64, 3, 32), (1, 60, 64, 64, 8),
                                                        (1, 90, 128, 4, 16), (1, 60, 136, 4, 16),
                                                        (1, 237, 136, 4, 16), (1, 240, 136, 4, 16), (2, 171, 136, 4, 16),
                                                        (1, 5, 64, 5, 16), (1, 97, 64, 9, 8), (1, 139, 40, 3, 24),
                                                        (1, 153, 64, 4, 16), (1, 154, 64, 4, 16), (1, 153, 200, 2, 32), (1, 155, 136, 2, 24)])
def test_attention_projection(cuda_device, batch, n, c_z, heads, head_dim):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n + heads)
    params = orc.round_params(orc.random_triatt_params(rng, c_z=c_z, heads=heads, c_hidden=head_dim, std=0.1, ln_noise=0.1), "bfloat16")
    x = orc.round_bf16(rng.standard_normal((batch, n, n, c_z)).astype(np.float32))
    mask = np.ones((batch, n, n), np.float32)
    got = triangle_attention_forward(params, x, mask, starting=False, dtype="bfloat16")
    _lib.device_status()
    assert_parity(orc.triangle_attention(params, x, mask, False, dtype="bfloat16"), got, label=f"{batch} x {n} {c_z} {heads}x{head_dim}")
