"""The general path's bf16 attention core: one to five steps of 64 keys, four rows to an item and three
(by how many rounds of items each needs), two for wide heads, rows past the last group, scores that rise
by more than the offset may lag behind, rows without a kept key (whose offsets lie beyond the integers
that floats hold) and items of one step, where the next item's scores follow at once.

Tolerance: the benchmark's bf16 budget (conftest.assert_parity), which takes scores of a few units: where
two roundings of q or k differ by an ulp (2^-9 of values up to 3), scores of a deviation s differ by up to
2^-7 s, and so do weights. At std = 0.2 that is 0.02 of single weights (s = 2.6)."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,heads,head_dim,std", [
    (17, 4, 16, 0.1), (64, 12, 32, 0.1),   # one step
    (65, 4, 16, 0.1), (100, 12, 32, 0.1),  # two steps; three rows to an item
    (130, 4, 16, 0.2), (193, 8, 24, 0.1),  # three, with larger scores; four steps
    (129, 2, 64, 0.2), (257, 4, 16, 0.1),  # wide heads, two rows; five steps
    (70, 4, 8, 0.1), (131, 6, 8, 0.2),     # heads that fill half a tile of 16
])
def test_general_core(cuda_device, n, heads, head_dim, std):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n + heads)
    c_z = 64
    params = orc.round_params(orc.random_triatt_params(rng, c_z=c_z, heads=heads, c_hidden=head_dim, std=std, ln_noise=0.1), "bfloat16")
    x = orc.round_bf16(rng.standard_normal((1, n, n, c_z)).astype(np.float32))
    mask = orc.pad_mask(n, n // 9)
    mask[0, 3] = 0.0  # a row without a key
    mask[0, 5, : n // 2] = 0.0  # one whose first steps are dropped
    emu = orc.triangle_attention(params, x, mask, starting=True, dtype="bfloat16")
    got = triangle_attention_forward(params, x, mask, starting=True, dtype="bfloat16")
    _lib.device_status()
    kept = np.broadcast_to(mask.any(axis=2)[:, :, None, None], x.shape)
    assert_parity(emu, got, where=kept, label=f"general core n={n} {heads}x{head_dim}")
    # (the sum with -1e9 absorbs scores below 32)
    assert_parity(emu, got, where=~kept, label=f"general core n={n} {heads}x{head_dim}, rows without a key")
