"""Trailing dropped keys: one, several and most of the keys, ends inside and between steps of 64, rows of one item that
end differently, rows without a kept key (the average of all keys) beside others, soft and hard mask values mixed in a step, and
dropped keys that do count: beside scores as low as theirs, and by values that are not finite.

Tolerance: the benchmark's bf16 budget (conftest.assert_parity). Where dropped keys have no weight, the
bits are those of a call whose last key is kept, with a bias that leaves it no weight."""

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


def _padded(n_k, dropped, cuda_device):
    """Operands of 7 rows and 40 queries whose last keys are dropped, and the call."""
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import attention_core

    rng = np.random.default_rng(n_k + dropped)
    draw = lambda *shape, scale=1.0: orc.round_bf16(rng.normal(size=shape, scale=scale).astype(np.float32))
    q, k, v = draw(1, 7, 4, 40, 32, scale=0.5), draw(1, 7, 4, n_k, 32, scale=0.5), draw(1, 7, 4, n_k, 32)
    tb, mb = draw(1, 1, 4, 40, n_k), np.zeros((1, 7, 1, 1, n_k), np.float32)
    mb[..., n_k - dropped:] = -1e9

    def run():
        t = lambda a, dtype=torch.bfloat16: torch.from_numpy(a).to(cuda_device).to(dtype)
        out = attention_core(t(q), t(k), t(v), t(tb), t(mb, torch.float32))
        _lib.device_status()
        return out.float().cpu().numpy()

    return q, k, v, tb, mb, run


PADDED = [(257, 1), (321, 70), (512, 64), (512, 130), (640, 200), (1280, 81)]


@pytest.mark.parametrize("n_k,dropped", PADDED)
def test_dropped_keys_beside_low_scores(cuda_device, n_k, dropped):
    """A dropped key's score is -30000: it has weight beside kept keys that score no better, masked by the pair bias or by soft
    mask values, and then all dropped keys have it, in whichever step. The other queries' bits stay. (Scores near
    30000 are within 2^-8 of exact in float32, and so are weights; the parity budget allows five times that.)"""
    q, k, v, tb, mb, run = _padded(n_k, dropped, cuda_device)
    plain = run()
    tb[:, :, :, 3, : n_k - dropped] = -1e5  # every kept key of a query
    tb[:, :, :, 17, : n_k - dropped] -= 29952.0
    tb[:] = orc.round_bf16(tb)
    mb[:, 2, :, :, : n_k - dropped] = -29995.0  # every kept key of a row
    mb[:, 5, :, :, : 64] = -1e9  # nothing kept in the first step
    got = run()
    s = np.einsum("bihjd,bihkd->bihjk", q.astype(np.float64), k) + tb + mb
    s = np.where(mb <= -30000.0, -30000.0, s)
    w = np.exp(s - s.max(-1, keepdims=True))
    assert_parity(np.einsum("bihjk,bihkd->bihjd", w / w.sum(-1, keepdims=True), v), got, label=f"low scores, {n_k} keys, {dropped} dropped")
    same = np.ones_like(got, bool)
    same[:, [2, 5]] = same[:, :, :, [3, 17]] = False
    assert np.array_equal(got[same], plain[same])


@pytest.mark.parametrize("n_k,dropped", PADDED)
def test_dropped_values_that_are_not_finite(cuda_device, n_k, dropped):
    """A weight of zero times an infinity is not a number, in the reference as here, in whichever step."""
    _, _, v, _, _, run = _padded(n_k, dropped, cuda_device)
    plain = run()
    v[0, 1, 2, -1, 5], v[0, 4, 0, n_k - dropped, 31], v[0, 6, 3, -1, 0] = np.inf, np.nan, -np.inf
    got = run()
    gone = np.zeros_like(got, bool)
    gone[0, 1, 2, :, 5] = gone[0, 4, 0, :, 31] = gone[0, 6, 3, :, 0] = True
    assert np.isnan(got[gone]).all() and np.array_equal(got[~gone], plain[~gone])
