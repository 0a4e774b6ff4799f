"""The block's float32 single track (split-bf16 products on the tensor cores) at the sizes where
its tiles end: rows around 128, few heads, hidden widths that are no multiple of 8 or 64 (the
padded weight copy), weights TMA cannot read in place, and K split over several partial sums.

Given the pair tensor the block produced, the single track is recomputed in float64 on the same
bf16 weights. Tolerance 2e-4, the reference test's own for this op
(tests/models/boltz2/test_attention_checkpoint_parity.py:47-52); float32 sums over at most 1536
products of order one stay below 1536 * 2^-24 = 1e-4 of their scale."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _params(rng, heads, hidden):
    c_s = 24 * heads
    params = orc.random_pairformer_params(rng, c_s=c_s, heads_s=heads, std=0.05, ln_noise=0.1)
    w = lambda *shape: (rng.standard_normal(shape) * 0.05).astype(np.float32)
    params["transition_s"] = {"norm": params["transition_s"]["norm"], "fc1": {"kernel": w(c_s, hidden)},
                              "fc2": {"kernel": w(c_s, hidden)}, "fc3": {"kernel": w(hidden, c_s)}}
    return orc.round_params(params, "bfloat16")


def _misaligned(t):
    """The same values 2 bytes off a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


@pytest.mark.parametrize("n,heads,hidden,shift", [(1, 1, 8, False), (127, 4, 100, False), (129, 16, 1536, False),
                                                  (128, 16, 1537, True), (260, 3, 64, False), (40, 16, 36, True)])
def test_single_track_against_float64(cuda_device, n, heads, hidden, shift):
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.pairformer import pairformer_forward

    rng = np.random.default_rng(n + hidden)
    params = _params(rng, heads, hidden)
    z = orc.round_bf16(rng.standard_normal((1, n, n, 128)).astype(np.float32))
    s = rng.standard_normal((1, n, 24 * heads)).astype(np.float32)
    mask = (rng.random((1, n)) < 0.9).astype(np.float32)
    mask[0, 0] = 1.0
    pd = dev.params_to_device(params)
    if shift:
        for group, names in (("attention", ("proj_q", "proj_k", "proj_v", "proj_g", "proj_o")),
                             ("transition_s", ("fc1", "fc2", "fc3"))):
            for name in names:
                pd[group][name]["kernel"] = _misaligned(pd[group][name]["kernel"])
    s_got, z_got = pairformer_forward([pd], torch.from_numpy(s).cuda(), dev.to_device(z, torch.bfloat16),
                                      torch.from_numpy(mask).cuda(), torch.ones(1, n, n, device="cuda"))
    _lib.device_status()
    s_got, z_got = s_got.cpu().numpy(), z_got.float().cpu().numpy()
    sn = orc.layer_norm(s, params["pre_norm_s"]["scale"], params["pre_norm_s"]["bias"], 1e-5)
    ref = s + orc.attention_pair_bias(params["attention"], sn, z_got, mask, k_in=sn, dtype="float64")
    ref = ref + orc.transition(params["transition_s"], ref, dtype="float64")
    np.testing.assert_allclose(s_got, ref, rtol=2e-4, atol=2e-4)


@pytest.mark.parametrize("n,heads", [(1, 1), (40, 3), (129, 16)])
def test_single_representation_off_the_16_byte_grid(cuda_device, monkeypatch, n, heads):
    """Views that start one float past a 16-byte boundary, as input and as result: the same bits."""
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.attention import attention_pair_bias_forward
    from foldjax_b200.pairformer import pairformer_forward

    rng = np.random.default_rng(n)
    pd = dev.params_to_device(_params(rng, heads, 64))
    z = dev.to_device(rng.standard_normal((1, n, n, 128)).astype(np.float32), torch.bfloat16)
    s, k_in = (torch.from_numpy(rng.standard_normal((1, n, 24 * heads)).astype(np.float32)).cuda() for _ in range(2))
    mask = torch.ones(1, n, device="cuda")

    def run(move):
        return [attention_pair_bias_forward(pd["attention"], move(s), z, mask, k_in=move(k_in)),
                *pairformer_forward([pd, pd], move(s), z, mask, None)]

    want = run(lambda t: t)
    _lib.device_status()
    new = torch.empty_like
    monkeypatch.setattr(torch, "empty_like", lambda t: _misaligned(new(t)) if t.dtype == torch.float32 else new(t))
    got = run(_misaligned)
    _lib.device_status()
    assert got[0].data_ptr() % 16 and got[1].data_ptr() % 16
    for w, g in zip(want, got):
        assert torch.equal(w, g)


@pytest.mark.parametrize("limit", [40, 24])  # (16 heads x 2 tiles of queries: a CTA for each tile, and for two)
def test_results_do_not_depend_on_the_sm_limit(cuda_device, limit):
    """Fewer SMs, the same K splits and therefore the same bits."""
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.pairformer import pairformer_forward

    rng = np.random.default_rng(9)
    n, lib = 136, _lib.load()
    pd = dev.params_to_device(_params(rng, 16, 1536))
    z = dev.to_device(rng.standard_normal((1, n, n, 128)).astype(np.float32), torch.bfloat16)
    s = torch.from_numpy(rng.standard_normal((1, n, 384)).astype(np.float32)).cuda()
    want = pairformer_forward([pd, pd], s, z, torch.ones(1, n, device="cuda"), None)
    _lib.check(lib.b200tri_set_sm_limit(limit))
    try:
        got = pairformer_forward([pd, pd], s, z, torch.ones(1, n, device="cuda"), None)
        _lib.device_status()
    finally:
        _lib.check(lib.b200tri_set_sm_limit(0))
    for w, g in zip(want, got):
        assert torch.equal(w, g)


@pytest.mark.parametrize("n", [129, 150, 176, 250, 256, 257, 300, 385])
def test_two_tiles_of_queries_to_a_cta(cuda_device, n):
    """The attention's form for more tiles than SMs, at 7 SMs: even and odd numbers of tiles, whose last CTA of a head then has one that does
    not exist, several items a CTA, last steps of all widths. The bits of the form with a CTA for each tile, which the same
    call takes with all SMs."""
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.attention import attention_pair_bias_forward

    rng, lib = np.random.default_rng(n), _lib.load()
    params = orc.round_params(orc.random_attention_pair_bias_params(rng, c_s=384, heads=16, std=0.05, ln_noise=0.1), "bfloat16")
    s = rng.standard_normal((1, n, 384)).astype(np.float32)
    z = orc.round_bf16(rng.standard_normal((1, n, n, 128)).astype(np.float32))
    mask = (rng.random((1, n)) < 0.85).astype(np.float32)
    mask[0, -1] = 1.0
    args = (dev.params_to_device(params), torch.from_numpy(s).cuda(), dev.to_device(z, torch.bfloat16), torch.from_numpy(mask).cuda())
    want = attention_pair_bias_forward(*args)
    _lib.check(lib.b200tri_set_sm_limit(7))
    try:
        got = attention_pair_bias_forward(*args)
        _lib.device_status()
    finally:
        _lib.check(lib.b200tri_set_sm_limit(0))
    assert torch.equal(got, want)
    np.testing.assert_allclose(got.cpu().numpy(), orc.attention_pair_bias(params, s, z, mask, dtype="float64"), rtol=2e-4, atol=2e-4)
