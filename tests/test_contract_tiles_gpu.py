"""The contraction in tiles of 256 rows (large n_k): a last tile whose second half has one row, a
ragged one, or none, columns that end in partial blocks, one and two sources, bf16 results and
float32 running sums; a shape with small n_k takes tiles of 128 rows, and so do, with 128 columns, the two of no
more than 128 columns. Then the same tiles over operands and a result in blocks of 64 rows, as the fused
multiplication lays them out.

The float32 sum of m products is within m * 2^-23 of sum |a||b| of the exact one, however it is
rounded; bf16 results are rounded once more (2^-8 relative)."""

from __future__ import annotations

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_i,n_j,n_k,n_src", [(385, 513, 640, 2), (400, 40, 1000, 1), (521, 72, 1536, 1), (264, 300, 200, 1),
                                               (400, 140, 1000, 1), (400, 264, 1000, 1), (521, 140, 1536, 1), (521, 520, 1536, 1)])
@pytest.mark.parametrize("running", [False, True])
def test_contract(cuda_device, n_i, n_j, n_k, n_src, running):
    from foldjax_b200 import _lib, _device as dev

    torch.manual_seed(n_i + n_k)
    ld, ld_j = (n_k + 7) // 8 * 8, (n_j + 7) // 8 * 8
    a = torch.randn(n_src, 128, n_i, ld, device=cuda_device).bfloat16()
    b = torch.randn(n_src, 128, n_j, ld, device=cuda_device).bfloat16()
    a[..., n_k:] = b[..., n_k:] = 0
    ref = sum(s.double() @ t.double().mT for s, t in zip(a, b))
    bound = n_src * n_k * 2.0 ** -23 * sum(s.float().abs() @ t.float().abs().mT for s, t in zip(a, b))
    out = torch.full((128, n_i, ld_j), float("nan"), dtype=torch.float32 if running else torch.bfloat16, device=cuda_device)
    acc = torch.randn_like(out) if running else None
    args = _lib.TrimulContractArgs(
        n_i=n_i, n_j=n_j, n_k=n_k, n_src=n_src,
        a=a.data_ptr(), a_ld=ld, a_chan_stride=n_i * ld, a_src_stride=128 * n_i * ld,
        b=b.data_ptr(), b_ld=ld, b_chan_stride=n_j * ld, b_src_stride=128 * n_j * ld,
        acc_in=acc.data_ptr() if running else None, out_f32=out.data_ptr() if running else None,
        out_bf16=None if running else out.data_ptr(), out_ld=ld_j, out_chan_stride=n_i * ld_j,
    )
    _lib.check(_lib.load().b200tri_trimul_contract(C.byref(args), C.c_void_p(dev.stream_ptr())))
    _lib.device_status()
    if running:
        ref = ref + acc[..., :n_j].double()
        bound = bound + 2.0 ** -23 * ref.abs()
    else:
        bound = bound * 1.01 + 2.0 ** -8 * ref.abs()
    got = out[..., :n_j].double()
    assert bool(((got - ref).abs() <= bound).all())  # (false where a value was not written)
    assert bool(out[..., n_j:].isnan().all())  # the pitch padding stays as it was


def _blocked(rows, fill):
    """[..., rows, ld] -> [block][...][64][ld], the last block filled up with `fill`."""
    pad = -rows.shape[-2] % 64
    rows = torch.cat([rows, rows.new_full((*rows.shape[:-2], pad, rows.shape[-1]), fill)], -2)
    return torch.stack(rows.split(64, -2))


# (wide tiles but for the last shape: a last tile of 235 rows, of 132 and 129 (a second half of a few
# rows), of 32 and of 1 (an empty one). Rows of a multiple of 8 columns leave by TMA, others do not.)
@pytest.mark.parametrize("n_i,n_j,n_src", [(1003, 1003, 1), (1003, 1008, 1), (900, 1000, 1), (1153, 1160, 1), (800, 808, 1),
                                           (769, 776, 1), (700, 712, 2), (203, 208, 1)])
def test_contract_in_blocks_of_64_rows(cuda_device, n_i, n_j, n_src):
    from foldjax_b200 import _lib, _device as dev

    torch.manual_seed(n_i)
    n_k = n_i
    ld, ld_j = (n_k + 63) // 64 * 64, (n_j + 63) // 64 * 64
    nan, untouched = float("nan"), 12352.0
    # what lies past the rows, and past the k range of a row, is never read into a result
    plain = [torch.randn(n_src, 128, n, n_k, device=cuda_device).bfloat16() for n in (n_i, n_j)]
    a, b = (torch.stack([_blocked(torch.nn.functional.pad(s, (0, ld - n_k), value=nan), nan) for s in side]) for side in plain)
    ref = sum(s.double() @ t.double().mT for s, t in zip(*plain))
    bound = n_src * n_k * 2.0 ** -23 * sum(s.float().abs() @ t.float().abs().mT for s, t in zip(*plain)).double()
    blocks = a.shape[1]
    out = torch.full((blocks, 128, 64, ld_j), untouched, dtype=torch.bfloat16, device=cuda_device)
    chan, block = 64 * ld, 128 * 64 * ld
    args = _lib.TrimulContractArgs(
        n_i=n_i, n_j=n_j, n_k=n_k, n_src=n_src,
        a=a.data_ptr(), a_ld=ld, a_chan_stride=chan, a_src_stride=blocks * block, a_rows_per_block=64, a_block_stride=block,
        b=b.data_ptr(), b_ld=ld, b_chan_stride=chan, b_src_stride=b.shape[1] * block, b_rows_per_block=64, b_block_stride=block,
        out_bf16=out.data_ptr(), out_ld=ld_j, out_chan_stride=64 * ld_j, out_rows_per_block=64, out_block_stride=128 * 64 * ld_j,
    )
    _lib.check(_lib.load().b200tri_trimul_contract(C.byref(args), C.c_void_p(dev.stream_ptr())))
    _lib.device_status()
    rows = out.transpose(0, 1).reshape(128, blocks * 64, ld_j)
    got = rows[:, :n_i, :n_j].double()
    assert bool(((got - ref).abs() <= bound * 1.01 + 2.0 ** -8 * ref.abs()).all())
    assert bool((rows[:, n_i:] == untouched).all()) and bool((rows[:, :n_i, n_j:] == untouched).all())
