"""The same operator on two streams, and from two threads, at once, and captured
in graphs: every call gets the bits it gets alone. Sizes differ, so that shared scratch would show in
either direction."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from oracle import triangle_oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _calls(device):
    """name -> (function of a pair tensor and mask), all entry points that take scratch."""
    from foldjax_b200 import _device as dev
    from foldjax_b200.pairformer import pairformer_forward
    from foldjax_b200.transition import transition_forward
    from foldjax_b200.triangle import triangle_multiplication_forward
    from foldjax_b200.triangle_attention import attention_core, triangle_attention_forward

    rng = np.random.default_rng(3)
    block = dev.params_to_device(orc.random_pairformer_params(rng, std=0.05, ln_noise=0.1))
    f32 = dev.params_to_device(orc.random_triatt_params(rng, std=0.05, ln_noise=0.1), torch.float32)

    def core(z, m):
        n = z.shape[1]
        q = z[..., :128].reshape(1, n, n, 4, 32).permute(0, 1, 3, 2, 4).contiguous()
        return attention_core(q, q, q, z[..., :4].permute(0, 3, 1, 2)[:, None].contiguous(),
                              (1e9 * (m - 1))[:, :, None, None, :])

    def trunk(z, m):
        s = z[:, :, 0, :].float().repeat(1, 1, 3).contiguous()
        return torch.cat([t.float().reshape(-1) for t in pairformer_forward([block, block], s, z, m[:, 0].contiguous(), m)])

    return {
        "mul": lambda z, m: triangle_multiplication_forward(block["tri_mul_out"], z, m, "outgoing", residual=z),
        "attn": lambda z, m: triangle_attention_forward(block["tri_att_end"], z, m, starting=False, residual=z),
        "attn f32": lambda z, m: triangle_attention_forward(f32, z.float(), m),
        "transition": lambda z, m: transition_forward(block["transition_z"], z, residual=z),
        "core": core,
        "trunk": trunk,
    }


def _inputs(device, sizes):
    g = torch.Generator(device=device).manual_seed(5)
    out = []
    for n in sizes:
        z = torch.randn(1, n, n, 128, generator=g, device=device).bfloat16()
        m = (torch.rand(1, n, n, generator=g, device=device) > 0.1).float()
        m[..., 0] = 1.0
        out.append((z, m))
    return out


CALLS = [(name, (200, 136, 264)) for name in ("mul", "attn", "attn f32", "transition", "core", "trunk")]
CALLS += [("core", (60, 48, 64))]  # (whose first kernel is launched programmatically)


@pytest.mark.parametrize("name,sizes", CALLS)
@pytest.mark.parametrize("threads", [False, True])
def test_concurrent_calls_equal_calls_one_by_one(cuda_device, name, sizes, threads):
    from foldjax_b200 import _lib

    call = _calls(cuda_device)[name]
    inputs = _inputs(cuda_device, sizes[:2])
    want = [call(z, m) for z, m in inputs]
    torch.cuda.synchronize()
    got = [[] for _ in inputs]
    repeats = 12
    # two streams fed in turn by one thread, or one stream fed by two threads
    streams = [torch.cuda.Stream() for _ in range(1 if threads else 2)]

    def feed(i, count):
        with torch.cuda.stream(streams[i % len(streams)]):
            for _ in range(count):
                got[i].append(call(*inputs[i]))

    if threads:
        workers = [threading.Thread(target=feed, args=(i, repeats)) for i in range(2)]
        for w in workers:
            w.start()
        for w in workers:
            w.join()
    else:
        for _ in range(repeats):
            for i in range(2):
                feed(i, 1)
    torch.cuda.synchronize()
    _lib.device_status()
    for w, results in zip(want, got):
        assert len(results) == repeats
        for r in results:
            assert torch.equal(r, w)


@pytest.mark.parametrize("name,sizes", CALLS)
def test_captured_calls(cuda_device, name, sizes):
    """Two graphs captured on one stream, replayed on two, while eager calls of a larger size run and
    the kept scratch is dropped."""
    from foldjax_b200 import _device as dev, _lib

    call = _calls(cuda_device)[name]
    inputs = _inputs(cuda_device, sizes)
    want = [call(z, m) for z, m in inputs]
    torch.cuda.synchronize()
    capture, graphs = torch.cuda.Stream(), []
    with torch.cuda.stream(capture):
        call(*inputs[1])
    torch.cuda.synchronize()
    for z, m in inputs[:2]:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=capture):
            out = call(z, m)
        graphs.append((graph, out))
    dev.release_workspaces()
    streams = [torch.cuda.Stream() for _ in graphs]
    eager = []
    for _ in range(4):
        for (graph, _), stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
        eager.append(call(*inputs[2]))
    torch.cuda.synchronize()
    _lib.device_status()
    for (_, out), w in zip(graphs, want):
        assert torch.equal(out, w)
    for e in eager:
        assert torch.equal(e, want[2])
