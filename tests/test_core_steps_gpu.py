"""The attention core's walk over the keys in steps of 64: remainders of the last step, maxima that rise
from step to step (the running state is rescaled), first keys that are dropped, scores far below the
maximum, and row counts around its groups of rows."""

import numpy as np
import pytest
import torch

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_i,n_k", [(1, 1), (3, 31), (4, 32), (5, 33), (2, 63), (1, 64), (7, 96), (4, 97), (3, 130), (9, 225)])
@pytest.mark.parametrize("bias", ["flat", "rising", "falling", "first_dropped"])
def test_core_steps(cuda_device, n_i, n_k, bias):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import attention_core

    n_j = 131
    rng = np.random.default_rng(100 * n_i + n_k)
    draw = lambda *shape, scale=1.0: orc.round_bf16(rng.normal(size=shape, scale=scale).astype(np.float32))
    q, k, v = draw(1, n_i, 4, n_j, 32, scale=0.5), draw(1, n_i, 4, n_k, 32, scale=0.5), draw(1, n_i, 4, n_k, 32)
    tb = draw(1, 1, 4, n_j, n_k)
    mb = np.zeros((1, n_i, 1, 1, n_k), np.float32)
    half_step = np.arange(n_k) // 32
    if bias == "rising":  # by more than the 2^8 that P may grow, in every half step
        tb = orc.round_bf16(tb + 12.0 * half_step.astype(np.float32))
    elif bias == "falling":  # to scores that no longer count
        tb = orc.round_bf16(tb - 200.0 * half_step.astype(np.float32))
    elif bias == "first_dropped":
        mb[..., : min(40, n_k - 1)] = -1e9
    ref = orc.attention_core(q, k, v, tb, mb, dtype="bfloat16")
    t = lambda a, dtype=torch.bfloat16: torch.from_numpy(a).to(cuda_device).to(dtype)
    got = attention_core(t(q), t(k), t(v), t(tb), t(mb, torch.float32))
    _lib.device_status()
    assert_parity(ref, got.float().cpu().numpy(), label=f"core steps {n_i}x{n_k} {bias}")
