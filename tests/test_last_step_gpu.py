"""The attention cores' last step of keys, of which 16, 32, 48 or all 64 columns are computed: remainders at the edges
of these widths, as the only step, behind a whole one and behind several, with rows that keep no key (whose weights show a column too
many or too few) and with scores that reach their maximum in the last step. 48 columns are taken by the 128-channel core where there
is no whole step or more than one, by the float32 core for heads of up to 32 in up to two steps, and by the general
bf16 core for heads of up to 32; elsewhere those keys take 64. With three SMs a CTA goes on from a short last step to its next items.

Tolerances are those of the other tests of each core: the bf16 budget (conftest.assert_parity); float32 results of
order one against float64, 1e-4; the single track 2e-4 as in the reference's own test."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_parity
from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KEYS = [1, 15, 16, 17, 32, 33, 48, 49, 63, 80, 81, 96, 97, 112, 113, 128, 129, 144, 145, 160, 161, 176, 177, 192, 225, 240]


@pytest.mark.parametrize("n_k", KEYS)
def test_core(cuda_device, n_k):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import attention_core

    n_i, n_j = 5, 130
    rng = np.random.default_rng(n_k)
    draw = lambda *shape, scale=1.0: orc.round_bf16(rng.normal(size=shape, scale=scale).astype(np.float32))
    q, k, v = draw(1, n_i, 4, n_j, 32, scale=0.5), draw(1, n_i, 4, n_k, 32, scale=0.5), draw(1, n_i, 4, n_k, 32)
    tb = draw(1, 1, 4, n_j, n_k)
    tb[..., -1] += 14.0  # the last key moves the offset
    mb = np.zeros((1, n_i, 1, 1, n_k), np.float32)
    mb[:, 1] = -1e9
    mb[:, 2, ..., : n_k - 1] = -1e9
    tb = orc.round_bf16(tb)
    ref = orc.attention_core(q, k, v, tb, mb, dtype="bfloat16")
    t = lambda a, dtype=torch.bfloat16: torch.from_numpy(a).to(cuda_device).to(dtype)
    args = t(q), t(k), t(v), t(tb), t(mb, torch.float32)
    got, lib = attention_core(*args), _lib.load()
    _lib.check(lib.b200tri_set_sm_limit(3))  # (of 16 items)
    try:
        assert torch.equal(attention_core(*args), got)
        _lib.device_status()
    finally:
        _lib.check(lib.b200tri_set_sm_limit(0))
    assert_parity(ref, got.float().cpu().numpy(), label=f"core, {n_k} keys")


@pytest.mark.parametrize("n", [16, 17, 33, 48, 49, 80, 81, 96, 112, 113, 145, 161, 176])
@pytest.mark.parametrize("heads,head_dim,dtype", [(4, 16, "bfloat16"), (12, 32, "bfloat16"), (2, 64, "bfloat16"), (4, 32, "float32"),
                                                  (2, 64, "float32")])
def test_general_cores(cuda_device, n, heads, head_dim, dtype):
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n + heads)
    params = orc.random_triatt_params(rng, c_z=64, heads=heads, c_hidden=head_dim, std=0.1, ln_noise=0.1)
    x = rng.standard_normal((1, n, n, 64)).astype(np.float32)
    mask = orc.pad_mask(n, 1)
    mask[0, 3] = 0.0
    if dtype == "bfloat16":
        params, x = orc.round_params(params, dtype), orc.round_bf16(x)
    got = triangle_attention_forward(params, x, mask, starting=True, dtype=dtype)
    _lib.device_status()
    kept = np.broadcast_to(mask.any(axis=2)[:, :, None, None], x.shape)
    if dtype == "float32":
        ref = orc.triangle_attention(params, x, mask, starting=True, dtype="float64")
        assert np.abs(ref - got)[kept].max() <= 1e-4
        # (without a key float32 absorbs the scores under -1e9: a uniform average)
        ref = orc.triangle_attention(params, x, mask, starting=True, dtype="float32")
        assert np.abs(ref - got)[~kept].max() <= 1e-3
    else:
        ref = orc.triangle_attention(params, x, mask, starting=True, dtype="bfloat16")
        assert_parity(ref, got, where=kept, label=f"n={n} {heads}x{head_dim}")
        assert_parity(ref, got, where=~kept, label=f"n={n} {heads}x{head_dim}, rows without a key")


@pytest.mark.parametrize("n", [16, 17, 33, 48, 49, 80, 97, 113, 145, 161])
def test_single_track(cuda_device, n):
    from foldjax_b200 import _lib
    from foldjax_b200.attention import attention_pair_bias_forward

    rng = np.random.default_rng(n)
    params = orc.round_params(orc.random_attention_pair_bias_params(rng, c_s=384, heads=16, std=0.05, ln_noise=0.1), "bfloat16")
    s = rng.standard_normal((1, n, 384)).astype(np.float32)
    z = orc.round_bf16(rng.standard_normal((1, n, n, 128)).astype(np.float32))
    mask = (rng.random((1, n)) < 0.85).astype(np.float32)
    mask[0, -1] = 1.0
    got = attention_pair_bias_forward(params, s, z, mask)
    _lib.device_status()
    np.testing.assert_allclose(got, orc.attention_pair_bias(params, s, z, mask, dtype="float64"), rtol=2e-4, atol=2e-4)
