"""The kernels read the linear weights in place through TMA, which needs 16-byte alignment;
a weight that lies elsewhere goes through an aligned copy. Same values, so same bits."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _shifted(node):
    if isinstance(node, dict):
        return {k: _shifted(v) for k, v in node.items()}
    buf = torch.empty(node.numel() + 3, dtype=node.dtype, device=node.device)
    buf[3:] = node.reshape(-1)
    return buf[3:].view(node.shape)


@pytest.mark.parametrize("n", [1, 65, 130])
def test_weights_off_the_16_byte_grid(cuda_device, n):
    from foldjax_b200 import _device as dev
    from foldjax_b200.transition import transition_forward
    from foldjax_b200.triangle import triangle_multiplication_forward
    from foldjax_b200.triangle_attention import triangle_attention_forward

    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.standard_normal((n, n, 128)).astype(np.float32)).cuda().bfloat16()
    pm = dev.params_to_device(orc.random_trimul_params(rng, ln_noise=0.1))
    pa = dev.params_to_device(orc.random_triatt_params(rng, ln_noise=0.1))
    pt = dev.params_to_device(orc.random_transition_params(rng, ln_noise=0.1))
    assert torch.equal(triangle_multiplication_forward(pm, x, None, "incoming"),
                       triangle_multiplication_forward(_shifted(pm), x, None, "incoming"))
    assert torch.equal(triangle_attention_forward(pa, x), triangle_attention_forward(_shifted(pa), x))
    assert torch.equal(transition_forward(pt, x), transition_forward(_shifted(pt), x))
