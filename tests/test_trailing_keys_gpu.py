"""Trailing dropped keys, whose steps of 64 the attention core leaves out: one, several and more of them than
it looks at, sizes at which it does not look, ends inside and between steps, rows of one item that end differently, rows without a kept
key (the average of all keys) beside others, soft and hard mask values mixed in a step.

Tolerance: the benchmark's bf16 budget (conftest.assert_parity). Where nothing but zeros is left out, the
bits are those of a call that walks all steps: its last key is kept, with a bias that leaves it no weight."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


def _ends(n_i, n_k, dropped):
    """Per row: how many keys come before the trailing dropped ones."""
    ends = np.full(n_i, n_k - dropped)
    ends[4::7] = n_k - dropped - 64 if n_k - dropped > 64 else 1  # rows of one item that end differently
    ends[5::11] = 0                                               # rows without a kept key
    return ends


@pytest.mark.parametrize("n_k,dropped", [(193, 1), (200, 9), (256, 64), (257, 65), (321, 200), (449, 1), (512, 64), (513, 130), (513, 320), (640, 639),
                                           (1280, 81), (1281, 130)])
def test_core(cuda_device, n_k, dropped):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import attention_core

    n_i, n_j = 13, 40
    rng = np.random.default_rng(n_k + dropped)
    draw = lambda *shape, scale=1.0: orc.round_bf16(rng.normal(size=shape, scale=scale).astype(np.float32))
    q, k, v = draw(1, n_i, 4, n_j, 32, scale=0.5), draw(1, n_i, 4, n_k, 32, scale=0.5), draw(1, n_i, 4, n_k, 32)
    tb = draw(1, 1, 4, n_j, n_k)
    mb = np.zeros((1, n_i, 1, 1, n_k), np.float32)
    for i, end in enumerate(_ends(n_i, n_k, dropped)):
        mb[0, i, 0, 0, end:] = -1e9
    mb[0, 1, 0, 0, : n_k // 3 : 5] = -1e9  # dropped keys between kept ones
    mb[0, 2, 0, 0, : n_k // 3 : 3] = -2.5  # soft ones
    t = lambda a, dtype=torch.bfloat16: torch.from_numpy(a).to(cuda_device).to(dtype)
    got = attention_core(t(q), t(k), t(v), t(tb), t(mb, torch.float32))
    _lib.device_status()
    ref = orc.attention_core(q, k, v, tb, mb, dtype="bfloat16")
    assert_parity(ref, got.float().cpu().numpy(), label=f"trailing keys {n_k}, {dropped} dropped")
    some = np.flatnonzero((mb[0, :, 0, 0] > -1e8).any(axis=1))
    tb[..., -1], mb[..., -1] = orc.round_bf16(np.float32(-9000.0)), 0.0  # kept, without weight
    whole = attention_core(t(q), t(k), t(v), t(tb), t(mb, torch.float32))
    assert torch.equal(got[:, some], whole[:, some])
