"""Host-side argument checks that run before any kernel launch (no GPU needed).

The operators hand raw pointers to the kernels, so a result buffer of the wrong
size, dtype or layout must be refused in Python: on the device it would be a write
past the allocation."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

from foldjax_b200 import _device as dev


def test_out_buffer_must_match_the_input_exactly():
    like = torch.zeros(1, 8, 8, 128, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="shape"):
        dev.check_out(torch.zeros(1, 7, 8, 128, dtype=torch.bfloat16), like)
    with pytest.raises(ValueError, match="bfloat16"):
        dev.check_out(torch.zeros(1, 8, 8, 128, dtype=torch.float32), like)
    with pytest.raises(ValueError, match="contiguous"):
        dev.check_out(torch.zeros(1, 8, 128, 8, dtype=torch.bfloat16).transpose(2, 3), like)
    with pytest.raises(ValueError, match="torch tensor"):
        dev.check_out([1, 2, 3], like)
    # right shape, dtype and layout, but host memory: the kernels cannot write there
    with pytest.raises(ValueError, match="CUDA tensor"):
        dev.check_out(torch.zeros(1, 8, 8, 128, dtype=torch.bfloat16), like)


def test_residual_shape_is_compared_with_the_input():
    like = torch.zeros(1, 8, 8, 128, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="residual shape"):
        dev.check_same_shape(torch.zeros(1, 4, 4, 128), like, "residual")
    assert dev.check_same_shape(like, like, "residual") is like


def test_workspace_reuse_accounts_for_the_alignment_slack(monkeypatch):
    """A cached buffer is reused only if it still covers the request after the pointer
    has been rounded up to 1 KiB."""
    real_empty = torch.empty

    def fake_empty(n, dtype=None, device=None):
        return real_empty(int(n), dtype=torch.uint8)

    monkeypatch.setattr(dev.torch, "empty", fake_empty)
    monkeypatch.setattr(dev.torch.cuda, "current_device", lambda: 0)
    dev.release_workspaces()
    a = dev.workspace(4096, "t")
    assert a.numel() == 4096 + 1024
    assert dev.workspace(4096, "t") is a
    assert dev.workspace(3000, "t") is a
    b = dev.workspace(4097, "t")  # 4097 + 1024 > 5120: the old buffer no longer covers it
    assert b is not a and b.numel() == 4097 + 1024
    dev.release_workspaces()


def _host_scratch(monkeypatch):
    """dev.workspace on host memory; returns the stream handle it sees, to be changed by the test."""
    real_empty, stream = torch.empty, [1]
    monkeypatch.setattr(dev.torch, "empty", lambda n, dtype=None, device=None: real_empty(int(n), dtype=torch.uint8))
    monkeypatch.setattr(dev.torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(dev.torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(dev.torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(dev, "stream_ptr", lambda: stream[0])
    dev.release_workspaces()
    return stream


def test_streams_do_not_share_scratch(monkeypatch):
    stream = _host_scratch(monkeypatch)
    a = dev.workspace(4096, "t")
    stream[0] = 2
    b = dev.workspace(4096, "t")
    assert a is not b and dev.workspace(4096, "t") is b
    stream[0] = 1
    assert dev.workspace(4096, "t") is a
    # a program that goes through many streams keeps the buffers of the last few
    for stream[0] in range(3, 2 + dev.STREAMS_KEPT):
        dev.workspace(4096, "t")
    stream[0] = 1
    assert dev.workspace(4096, "t") is a
    stream[0] = 2
    assert dev.workspace(4096, "t") is not b
    dev.release_workspaces()


def test_captured_calls_keep_no_scratch(monkeypatch):
    """A graph holds its buffers' addresses: nothing a later call can drop or write beside a replay."""
    _host_scratch(monkeypatch)
    kept = dev.workspace(4096, "t")
    monkeypatch.setattr(dev.torch.cuda, "is_current_stream_capturing", lambda: True)
    a = dev.workspace(4096, "t", (0, 1))
    b = dev.workspace(4096, "t", (0, 1))
    assert a is not kept and b is not kept and a is not b
    monkeypatch.setattr(dev.torch.cuda, "is_current_stream_capturing", lambda: False)
    assert dev.workspace(4096, "t") is kept
    dev.release_workspaces()


def test_exchange_scratch_is_held_by_the_op(monkeypatch):
    """A captured call's buffer is kept by nobody else: its pointer alone would outlive it."""
    from types import SimpleNamespace

    from foldjax_b200 import _lib, cp

    _host_scratch(monkeypatch)
    monkeypatch.setattr(dev.torch.cuda, "is_current_stream_capturing", lambda: True)
    size = SimpleNamespace(b200tri_trimul_cp_workspace_bytes=lambda *_: 4096, b200tri_triatt_cp_workspace_bytes=lambda *_: 8192)
    monkeypatch.setattr(_lib, "load", lambda: size)
    monkeypatch.setattr(cp, "TRANSPORT", "nccl")
    buf, pointer, nbytes = cp._exchange_workspace(SimpleNamespace(comm=0), 64)
    assert nbytes == 8192 and pointer % 1024 == 0
    assert buf.data_ptr() <= pointer and pointer + nbytes <= buf.data_ptr() + buf.numel()


def test_threads_do_not_share_scratch(monkeypatch):
    import gc
    import threading
    import weakref

    _host_scratch(monkeypatch)
    mine = dev.workspace(4096, "t")
    seen = []

    def other():
        buf = dev.workspace(4096, "t")
        assert buf is not mine and dev.workspace(4096, "t") is buf
        seen.append(weakref.ref(buf))

    thread = threading.Thread(target=other)
    thread.start()
    thread.join()
    gc.collect()
    assert seen and seen[0]() is None  # given back with the thread
    assert dev.workspace(4096, "t") is mine
    dev.release_workspaces()


def test_streamed_blocks_refuse_mismatched_host_buffers():
    """stream_host_blocks checks its host buffers before it touches a device."""
    from foldjax_b200.block import stream_host_blocks

    z = torch.zeros(1, 8, 8, 128, dtype=torch.bfloat16)
    run = lambda zd, md: zd + 1  # never reached
    assert stream_host_blocks(run, []) == []
    with pytest.raises(ValueError, match="bfloat16"):
        stream_host_blocks(run, [(z.float(), None)], [z.clone()])
    with pytest.raises(ValueError, match="same shape"):
        stream_host_blocks(run, [(z, None), (z[:, :4].contiguous(), None)], [z.clone(), z.clone()])
    with pytest.raises(ValueError, match="float32"):
        stream_host_blocks(run, [(z, torch.ones(1, 8, 8, dtype=torch.float64))], [z.clone()])
    with pytest.raises(ValueError, match="1 items but 2"):
        stream_host_blocks(run, [(z, None)], [z.clone(), z.clone()])
    with pytest.raises(ValueError, match="outputs must be"):
        stream_host_blocks(run, [(z, None)], [z.float()])


def test_block_variant_names_are_checked_before_any_device_work():
    from foldjax_b200.pairformer import VARIANTS, pairformer_forward

    assert set(VARIANTS) == {"boltz2", "protenix", "openfold3"}
    z = torch.zeros(1, 8, 8, 128, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="Unsupported pairformer variant"):
        pairformer_forward([{}], None, z, None, None, variant="alphafold2")


def test_pairformer_workspace_is_that_of_the_widest_block():
    """The blocks of a list may have transitions of different widths, and all use the same scratch: a
    workspace that only holds the first block's is refused before anything is launched."""
    import ctypes as C

    from foldjax_b200 import _lib

    lib = _lib.load()
    blocks = (_lib.PairformerBlockParams * 2)()
    for block, (hidden_z, hidden_s) in zip(blocks, [(512, 384), (256, 1536)]):
        block.transition_z.hidden, block.transition_s.hidden = hidden_z, hidden_s
    first, widest = (lib.b200tri_pairformer_workspace_bytes(64, 384, 16, 512, h) for h in (384, 1536))
    assert first < widest
    address = 1 << 20  # (never dereferenced: the call is refused)
    args = _lib.PairformerArgs(n=64, c_s=384, heads_s=16, n_blocks=2, params=blocks, z_in=address, z_out=address, s_in=address,
                               s_out=address, workspace=address, workspace_bytes=widest - 1025)
    assert lib.b200tri_pairformer_forward(C.byref(args), None) == _lib.ERR_WORKSPACE


def test_sm_reserves_add_up():
    """An inner reserve must not hand out the SMs that the one around it keeps free."""
    import ctypes as C

    from foldjax_b200 import _lib

    lib = _lib.load()
    # (C++ of the library's own: b200::sm_count, and b200::SmReserve's constructor and destructor)
    count, reserve, release = (getattr(lib, name) for name in ("_ZN4b2008sm_countEv", "_ZN4b2009SmReserveC1Ei", "_ZN4b2009SmReserveD1Ev"))
    reserve.argtypes, reserve.restype, release.argtypes, release.restype = [C.c_void_p, C.c_int], None, [C.c_void_p], None
    outer, inner = C.create_string_buffer(64), C.create_string_buffer(64)
    sms = count()
    for keep_outer, keep_inner in ((8, 5), (4, 100), (6, 0)):
        reserve(outer, keep_outer)
        assert count() == sms - keep_outer
        reserve(inner, keep_inner)
        assert count() == sms - keep_outer - keep_inner
        release(inner)
        assert count() == sms - keep_outer
        release(outer)
        assert count() == sms


def test_pairformer_needs_no_second_buffer_for_z():
    """What a stack of few tokens can make use of beyond the scratch of a block is not asked of a caller:
    scratch that was sized for a block is enough, and the single track's share grows with the tokens."""
    from foldjax_b200 import _lib

    lib = _lib.load()
    block = {n: lib.b200tri_pairformer_workspace_bytes(n, 384, 16, 512, 1536) for n in range(100, 140)}
    single = [block[n] - lib.b200tri_pairformer_workspace_bytes(n, 0, 0, 512, 0) for n in block]
    assert single == sorted(single)
    for n, least in block.items():
        more = lib.b200tri_pairformer_stack_workspace_bytes(n, 384, 16, 512, 1536, 48) - least
        assert more == (-(-n * n * 256 // 1024) * 1024 if n <= 128 else 0)
        assert lib.b200tri_pairformer_stack_workspace_bytes(n, 384, 16, 512, 1536, 1) == least
    assert lib.b200tri_pairformer_stack_workspace_bytes(64, 0, 0, 512, 0, 48) == lib.b200tri_pairformer_workspace_bytes(64, 0, 0, 512, 0)
    assert lib.b200tri_pairformer_stack_workspace_bytes(0, 384, 16, 512, 1536, 48) == 0


@pytest.mark.parametrize("stacked", [False, True])
@pytest.mark.parametrize("path,shape", [
    (("tri_mul_out", "p_in", "kernel"), (128, 128)), (("tri_att_end", "linear", "kernel"), (128, 3)),
    (("transition_z", "fc3", "kernel"), (256, 128)), (("transition_s", "fc2", "kernel"), (48, 96)),
    (("attention", "proj_q", "bias"), (24,)), (("transition_s", "norm", "scale"), (47,))])
def test_pairformer_parameters_of_another_shape_are_refused(monkeypatch, stacked, path, shape):
    """A block's parameters go to the kernels as bare pointers, so their shapes are compared first."""
    import numpy as np

    from foldjax_b200 import _lib
    from foldjax_b200.pairformer import pairformer_forward
    from oracle import triangle_oracle as orc

    class Reached(Exception):
        pass

    def reached(*_):
        raise Reached

    monkeypatch.setattr(dev, "require_cuda", lambda: None)
    monkeypatch.setattr(dev, "to_device", lambda x, dtype=None, device=None: torch.as_tensor(x).to(dtype).contiguous())
    monkeypatch.setattr(_lib, "workspace_bytes", reached)
    blocks = 3
    params = orc.random_pairformer_params(np.random.default_rng(0), c_s=48, heads_s=2)

    def lead(node):
        return {k: lead(v) for k, v in node.items()} if isinstance(node, dict) else np.stack([node] * blocks)

    def call(p, n=blocks):
        args = (torch.zeros(1, 8, 48), torch.zeros(1, 8, 8, 128), torch.ones(1, 8), torch.ones(1, 8, 8))
        return pairformer_forward(p, *args, num_blocks=n) if stacked else pairformer_forward([p], *args)

    good = lead(params) if stacked else params
    with pytest.raises(Reached):
        call(good)
    if stacked:
        with pytest.raises(Reached):
            call(good, blocks - 1)  # the first layers of a longer stack
        with pytest.raises(ValueError, match="behind an axis of 4 layers"):
            call(good, blocks + 1)
    node = good
    for key in path[:-1]:
        node = node[key]
    node[path[-1]] = np.zeros((blocks,) * stacked + shape, np.float32)
    with pytest.raises(ValueError, match=".".join(path)):
        call(good)


@pytest.mark.parametrize("gate", [0, 1])
def test_pairformer_refuses_a_pair_tensor_off_the_16_byte_grid(gate):
    """Before its first launch: the pair gate reads 16 bytes at a time."""
    import ctypes as C

    from foldjax_b200 import _lib

    lib = _lib.load()
    blocks = (_lib.PairformerBlockParams * 1)()
    blocks[0].transition_z.hidden = 512
    address = 1 << 20  # (never dereferenced)
    size = lib.b200tri_pairformer_workspace_bytes(64, 0, 0, 512, 0)
    for z_in, z_out in ((address + 2, address), (address, address + 8)):
        args = _lib.PairformerArgs(n=64, n_blocks=1, params=blocks, z_in=z_in, z_out=z_out, pair_mask=address, pair_gate=gate,
                                   workspace=address, workspace_bytes=size)
        assert lib.b200tri_pairformer_forward(C.byref(args), None) == _lib.ERR_INVALID
        assert b"16-byte aligned" in lib.b200tri_last_error()


def test_float32_attention_scratch_holds_nothing_twice():
    """Per pair and channel: the normalised row, q, k and v as three bf16 pieces each and the float32
    output; the gated output's pieces take the place of q's."""
    from foldjax_b200 import _lib

    n, c = 1024, 128
    size = _lib.load().b200tri_triatt_workspace_bytes_shape(n, _lib.DTYPE_F32, c, 4, 32)
    rows = n * n * c * (4 * 3 * 2 + 4)
    assert rows < size < 1.01 * rows
