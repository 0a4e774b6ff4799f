"""The general path's epilogues move 32 bytes at a time where rows lie on that grid: tensors that are
16 bytes off it, and channel and head counts whose rows cannot, give the bits of the aligned ones."""

import ctypes as C

import numpy as np
import pytest
import torch

from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu


def _off_by_16_bytes(x):
    skip = 16 // x.element_size()
    buf = torch.empty(x.numel() + 2 * skip, dtype=x.dtype, device=x.device)
    first = skip if buf.data_ptr() % 32 == 0 else 0
    view = buf[first:first + x.numel()].view(x.shape)
    view.copy_(x)
    assert view.data_ptr() % 32 == 16
    return view


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,c_z,c_hidden,heads,head_dim", [(37, 64, 128, 4, 16), (65, 72, 40, 3, 8), (33, 128, 72, 3, 24)])
def test_sixteen_bytes_off_the_sector_grid(cuda_device, dtype, n, c_z, c_hidden, heads, head_dim):
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.triangle import triangle_multiplication_forward
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n)
    pm = dev.params_to_device(orc.random_trimul_params(rng, c_z=c_z, c_hidden=c_hidden, std=0.1), dtype)
    pa = dev.params_to_device(orc.random_triatt_params(rng, c_z=c_z, heads=heads, c_hidden=head_dim, std=0.1), dtype)
    x = torch.randn(n, n, c_z, device="cuda").to(dtype)
    xs, out = _off_by_16_bytes(x), _off_by_16_bytes(torch.zeros_like(x))
    for direction in ("outgoing", "incoming"):
        assert torch.equal(triangle_multiplication_forward(pm, x, None, direction, residual=x),
                           triangle_multiplication_forward(pm, xs, None, direction, residual=xs, out=out))
    for starting in (True, False):
        assert torch.equal(triangle_attention_forward(pa, x, starting=starting, residual=x),
                           triangle_attention_forward(pa, xs, starting=starting, residual=xs, out=out))
    _lib.device_status()


@pytest.mark.parametrize("n_k", [64, 100])
def test_attention_operator_off_the_sector_grid(cuda_device, n_k):
    """Operands of the attention operator 16 bytes off: same bits."""
    from foldjax_b200 import _lib
    from foldjax_b200.triangle_attention import attention_core

    g = torch.Generator("cuda").manual_seed(n_k)
    q, k, v = (torch.randn(1, 5, 4, n, 32, generator=g, device="cuda").bfloat16() * 0.3 for n in (70, n_k, n_k))
    bias = torch.randn(1, 1, 4, 70, n_k, generator=g, device="cuda").bfloat16()
    mask = torch.zeros(1, 5, 1, 1, n_k, device="cuda")
    ref = attention_core(q, k, v, bias, mask)
    got = attention_core(*(_off_by_16_bytes(t) for t in (q, k, v, bias)), mask)
    _lib.device_status()
    assert torch.equal(ref, got)


def test_core_result_off_the_sector_grid(cuda_device):
    """The attention core's C entry with its result on and 16 bytes off the 32-byte grid: same bits."""
    from foldjax_b200 import _device as dev, _lib

    lib = _lib.load()
    n_i, n_j, n_k, h, d, ld = 5, 130, 70, 4, 32, 128
    g = torch.Generator("cuda").manual_seed(3)
    draw = lambda *shape, dtype=torch.bfloat16: (torch.randn(shape, generator=g, device="cuda") * 0.4).to(dtype)
    q, k, vt, bias = draw(n_i, n_j, h * d), draw(n_i, n_k, h * d), draw(n_i, h * d, ld, dtype=torch.float16), draw(h, n_j, ld)
    mask = torch.ones(n_i, n_k, device="cuda")
    nb = lib.b200tri_triatt_core_workspace_bytes(n_i, n_k)
    ws = torch.empty(nb + 1024, dtype=torch.uint8, device="cuda")
    on = torch.full((n_i, n_j, h * d), float("nan"), dtype=torch.bfloat16, device="cuda")
    off = _off_by_16_bytes(on)
    for o in (on, off):
        args = _lib.TriattCoreArgs(
            n_i=n_i, n_j=n_j, n_k=n_k, heads=h, head_dim=d, q=q.data_ptr(), k=k.data_ptr(), vt=vt.data_ptr(), v_ld=ld,
            bias=bias.data_ptr(), bias_ld=ld, bias_head_stride=n_j * ld, mask=mask.data_ptr(), ms_i=n_k, ms_k=1, inf=1e9,
            o=o.data_ptr(), unnormalized=0, workspace=dev.aligned_ptr(ws), workspace_bytes=nb)
        _lib.check(lib.b200tri_triatt_core(C.byref(args), C.c_void_p(dev.stream_ptr())))
    _lib.device_status()
    assert bool(torch.isfinite(on.float()).all()) and torch.equal(on, off)


@pytest.mark.parametrize("n,blocks", [(16, 4), (128, 3), (128, 4), (129, 3)])
def test_stack_with_and_without_left_over_sms(cuda_device, n, blocks):
    """Up to 128 tokens the pair bias of a stack runs aside and blocks end in two buffers in turn:
    the bits of one call per block."""
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.pairformer import pairformer_forward, pairformer_layer_forward

    rng = np.random.default_rng(n + blocks)
    params = [dev.params_to_device(orc.random_pairformer_params(rng, std=0.03, ln_noise=0.1), torch.bfloat16)
              for _ in range(blocks)]
    z = torch.randn(1, n, n, 128, device="cuda").bfloat16()
    s = torch.randn(1, n, 384, device="cuda")
    mask = torch.ones(1, n, device="cuda")
    mask[:, n - n // 16:] = 0
    pair = (mask[:, :, None] * mask[:, None, :]).contiguous()
    s1, z1 = s, z
    for p in params:
        s1, z1 = pairformer_layer_forward(p, s1, z1, mask, pair)
    for _ in range(3):
        s2, z2 = pairformer_forward(params, s, z, mask, pair, num_blocks=blocks)
        assert torch.equal(z1, z2) and torch.equal(s1, s2)
    _lib.device_status()
