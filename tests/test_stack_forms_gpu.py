"""Stacks of blocks of few tokens, where a block's pair bias runs beside the next block's pair track and blocks
end in two buffers in turn, through the C entry: every form gives the bits of one call per block."""

import ctypes as C

import numpy as np
import pytest

from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _inputs(n, blocks):
    from foldjax_b200 import _device as dev

    rng = np.random.default_rng(n + blocks)
    params = [dev.params_to_device(orc.random_pairformer_params(rng, std=0.03, ln_noise=0.1), torch.bfloat16)
              for _ in range(blocks)]
    g = torch.Generator("cuda").manual_seed(n)
    z = torch.randn(1, n, n, 128, generator=g, device="cuda").bfloat16()
    s = torch.randn(1, n, 384, generator=g, device="cuda")
    mask = torch.ones(1, n, device="cuda")
    mask[:, n - n // 16:] = 0
    return params, s, z, mask, (mask[:, :, None] * mask[:, None, :]).contiguous()


def _one_by_one(params, s, z, mask, pair, **flags):
    from foldjax_b200.pairformer import pairformer_forward

    for p in params:
        s, z = pairformer_forward([p], s, z, mask, pair, **flags)
    return s, z


def _in_one_call(params, s, z, mask, pair, stack_scratch=True, in_place=False, **flags):
    """b200tri_pairformer_forward with scratch for a block or for the stack, into new tensors or in place."""
    from foldjax_b200 import _device as dev, _lib
    from foldjax_b200.pairformer import _Packed

    lib, n, blocks = _lib.load(), z.shape[1], len(params)
    packed = [_Packed(p, True) for p in params]
    structs = (_lib.PairformerBlockParams * blocks).from_buffer_copy(b"".join(p.struct for p in packed))
    size = lib.b200tri_pairformer_workspace_bytes(n, 384, 16, packed[0].hidden_z, packed[0].hidden_s)
    if stack_scratch:
        size = lib.b200tri_pairformer_stack_workspace_bytes(n, 384, 16, packed[0].hidden_z, packed[0].hidden_s, blocks)
    size -= 1024  # (the reported sizes leave room to align the address)
    guard = 4096
    ws = torch.full((size + 1024 + guard,), 0xA5, dtype=torch.uint8, device="cuda")
    first = dev.aligned_ptr(ws) - ws.data_ptr()
    s, z = s.clone(), z.clone()
    s_out, z_out = (s, z) if in_place else (torch.empty_like(s), torch.empty_like(z))
    args = _lib.PairformerArgs(
        n=n, c_s=384, heads_s=16, n_blocks=blocks, stacked=0, eps=1e-5, tri_inf=1e9, att_inf=1e6, params=structs,
        z_in=z.data_ptr(), z_out=z_out.data_ptr(), s_in=s.data_ptr(), s_out=s_out.data_ptr(), pair_mask=pair.data_ptr(),
        mask=mask.data_ptr(), workspace=dev.aligned_ptr(ws), workspace_bytes=size, **{k: int(v) for k, v in flags.items()})
    _lib.check(lib.b200tri_pairformer_forward(C.byref(args), C.c_void_p(dev.stream_ptr())))
    _lib.device_status()
    assert bool((ws[first + size:] == 0xA5).all()) and bool((ws[:first] == 0xA5).all())
    return s_out, z_out


@pytest.mark.parametrize("n,blocks", [(16, 3), (100, 2), (128, 3), (129, 3)])
def test_scratch_for_a_block_is_enough_for_a_stack(cuda_device, n, blocks):
    inputs = _inputs(n, blocks)
    want = _one_by_one(*inputs)
    for stack_scratch in (False, True):
        got = _in_one_call(*inputs, stack_scratch=stack_scratch)
        assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


@pytest.mark.parametrize("n,blocks", [(40, 2), (100, 3), (128, 4)])
@pytest.mark.parametrize("flags", [{}, {"pair_gate": True}, {"mask_transition": True}, {"attention_first": True},
                                   {"pair_gate": True, "mask_transition": True, "attention_first": True}], ids=lambda f: "+".join(f) or "plain")
def test_stack_variants_and_in_place(cuda_device, n, blocks, flags):
    params, s, z, mask, pair = _inputs(n, blocks)
    # (dropped pairs that no token mask explains, so that the gate before the first update counts)
    pair = pair * (torch.rand(pair.shape, generator=torch.Generator("cuda").manual_seed(n), device="cuda") > 0.05)
    pair[0].fill_diagonal_(1.0)
    pair *= mask[:, :, None] * mask[:, None, :]
    want = _one_by_one(params, s, z, mask, pair, **flags)
    for in_place in (False, True):
        got = _in_one_call(params, s, z, mask, pair, in_place=in_place, **flags)
        assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


@pytest.mark.parametrize("threads", [False, True])
def test_stacks_at_once(cuda_device, threads):
    """Two streams fed by one thread, or two threads that feed one stream each: the side streams of the
    calls run beside one another."""
    import threading

    from foldjax_b200 import _lib
    from foldjax_b200.pairformer import pairformer_forward

    inputs = [_inputs(n, 4) for n in (100, 128)]
    want = [_one_by_one(*i) for i in inputs]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in inputs], [[] for _ in inputs]

    def feed(k, count):
        with torch.cuda.stream(streams[k]):
            got[k] += [pairformer_forward(*inputs[k]) for _ in range(count)]

    if threads:
        workers = [threading.Thread(target=feed, args=(k, 10)) for k in range(2)]
        for w in workers:
            w.start()
        for w in workers:
            w.join()
    else:
        for _ in range(10):
            for k in range(2):
                feed(k, 1)
    torch.cuda.synchronize()
    _lib.device_status()
    for w, results in zip(want, got):
        assert len(results) == 10 and all(torch.equal(w[0], s) and torch.equal(w[1], z) for s, z in results)


def test_captured_stack(cuda_device):
    """While a stream is captured the stack stays on it: replays beside an eager call, same bits."""
    from foldjax_b200 import _lib
    from foldjax_b200.pairformer import pairformer_forward

    captured, eager = _inputs(100, 3), _inputs(128, 3)
    want, beside = _one_by_one(*captured), _one_by_one(*eager)
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        pairformer_forward(*captured)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        s, z = pairformer_forward(*captured)
    for _ in range(3):
        with torch.cuda.stream(stream):
            graph.replay()
        s2, z2 = pairformer_forward(*eager)
        torch.cuda.synchronize()
        assert torch.equal(want[0], s) and torch.equal(want[1], z)
        assert torch.equal(beside[0], s2) and torch.equal(beside[1], z2)
    _lib.device_status()
