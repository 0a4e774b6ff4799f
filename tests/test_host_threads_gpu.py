"""Calls from host threads other than the one that loaded the library."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("op", ["transition", "mul", "attn"])
def test_first_call_of_a_thread(cuda_device, op):
    """A thread whose first call into CUDA is an operator of the library (with all memory it needs in
    the allocator's cache, nothing before it makes the device's context current)."""
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.transition import transition_forward
    from foldjax_b200.triangle import triangle_multiplication_forward
    from foldjax_b200.triangle_attention import triangle_attention_forward

    params = dev.params_to_device(orc.random_pairformer_params(np.random.default_rng(1), std=0.05))
    z = torch.randn(1, 40, 40, 128, device=cuda_device).bfloat16()
    call = {"transition": lambda: transition_forward(params["transition_z"], z),
            "mul": lambda: triangle_multiplication_forward(params["tri_mul_out"], z, None, "outgoing"),
            "attn": lambda: triangle_attention_forward(params["tri_att_start"], z)}[op]
    want = call()
    spare = call()
    del spare  # its memory serves the thread's call
    torch.cuda.synchronize()
    got = []

    def work():
        try:
            got.append(call())
        except Exception as error:  # noqa: BLE001 - reported below
            got.append(error)

    thread = threading.Thread(target=work)
    thread.start()
    thread.join()
    _lib.device_status()
    assert isinstance(got[0], torch.Tensor), got[0]
    assert torch.equal(got[0], want)
