"""BSR SpMM on block sizes and feature counts of both tensor-core kernels: block rows without blocks, fewer groups than
warps, odd numbers of groups, rows of more blocks than a warp keeps ids of, ragged slabs, an output that is not 16-byte aligned, calls of one wave
and of more."""
import numpy as np
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blk", [16, 32, 48, 64, 96])
@pytest.mark.parametrize("feat", [8, 64, 72, 176])
@pytest.mark.parametrize("counts", [[1], [0, 3, 0, 2, 5], [7, 1, 40]])
def test_matches_a_float64_product(cuda_device, blk, feat, counts):
    rng = np.random.default_rng(blk + feat + len(counts))
    nb, mb, nnzb = len(counts), 41, sum(counts)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(mb, k, replace=False)) for k in counts]).astype(np.int32)
    up = lambda x: torch.from_numpy(x).to(cuda_device)  # noqa: E731
    a = up(rng.standard_normal((nnzb, blk, blk)).astype(np.float16))
    b = up(rng.standard_normal((mb, blk, feat)).astype(np.float16))
    rows = torch.repeat_interleave(torch.arange(nb, device=cuda_device), up(np.diff(indptr)).long())
    ids = up(cols).long()
    want = torch.zeros(nb, blk, feat, dtype=torch.float64, device=cuda_device)
    mag = torch.zeros_like(want)
    want.index_add_(0, rows, torch.bmm(a.double(), b.double()[ids]))
    mag.index_add_(0, rows, torch.bmm(a.double().abs(), b.double().abs()[ids]))
    # fp32 sums of exact products; the tensor core may cut below the last bit once per 16 terms
    bound = mag * (max(counts) * blk / 16 + 8) * 2.0 ** -23
    for shift in (0, 1):
        c = torch.full((nb * blk * feat + 1,), 3.0, device=cuda_device)[shift:][:nb * blk * feat]
        ops.bsrmm(a.view(-1), b.view(-1), c, up(indptr), up(cols), nb, mb, nnzb, blk, feat)
        assert bool(((c.view(nb, blk, feat).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("blk", [16, 32, 48])
@pytest.mark.parametrize("feat", [64, 128, 136])
def test_rows_of_more_blocks_than_a_warp_keeps_ids_of(cuda_device, blk, feat):
    # a warp takes a quarter of a row's groups and reads the ids of its blocks 32 at a time: 31 to 34 and 75 blocks to a warp, from inside a block on
    # where a block is three groups
    rng = np.random.default_rng(blk + feat)
    counts, mb = [127, 0, 128, 129, 133, 300], 301
    nb, nnzb = len(counts), sum(counts)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(mb, k, replace=False)) for k in counts]).astype(np.int32)
    up = lambda x: torch.from_numpy(x).to(cuda_device)  # noqa: E731
    a = up(rng.standard_normal((nnzb, blk, blk)).astype(np.float16))
    b = up(rng.standard_normal((mb, blk, feat)).astype(np.float16))
    rows = torch.repeat_interleave(torch.arange(nb, device=cuda_device), up(np.diff(indptr)).long())
    want = torch.zeros(nb, blk, feat, dtype=torch.float64, device=cuda_device)
    mag = torch.zeros_like(want)
    want.index_add_(0, rows, torch.bmm(a.double(), b.double()[up(cols).long()]))
    mag.index_add_(0, rows, torch.bmm(a.double().abs(), b.double().abs()[up(cols).long()]))
    c = torch.full((nb * blk * feat,), 3.0, device=cuda_device)
    ops.bsrmm(a.view(-1), b.view(-1), c, up(indptr), up(cols), nb, mb, nnzb, blk, feat)
    bound = mag * (max(counts) * blk / 16 + 8) * 2.0 ** -23  # as above
    assert bool(((c.view(nb, blk, feat).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("nb,feat", [(1, 128), (100, 256), (101, 256), (60, 512), (296, 128), (297, 128), (148, 384), (149, 384), (98, 640), (3, 896)])
def test_blocks_of_32_on_either_side_of_a_wave(cuda_device, nb, feat):
    # thread blocks of one wave and more, items of one feature tile and of two, block rows without blocks
    rng = np.random.default_rng(nb + feat)
    blk, mb = 32, 17
    counts = rng.integers(0, 9, nb)
    counts[0] = 1
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(mb, k, replace=False)) for k in counts]).astype(np.int32)
    nnzb = len(cols)
    up = lambda x: torch.from_numpy(x).to(cuda_device)  # noqa: E731
    a = up(rng.standard_normal((nnzb, blk, blk)).astype(np.float16))
    b = up(rng.standard_normal((mb, blk, feat)).astype(np.float16))
    rows = torch.repeat_interleave(torch.arange(nb, device=cuda_device), up(counts).long())
    want = torch.zeros(nb, blk, feat, dtype=torch.float64, device=cuda_device)
    mag = torch.zeros_like(want)
    want.index_add_(0, rows, torch.bmm(a.double(), b.double()[up(cols).long()]))
    mag.index_add_(0, rows, torch.bmm(a.double().abs(), b.double().abs()[up(cols).long()]))
    c = torch.full((nb * blk * feat,), 3.0, device=cuda_device)
    ops.bsrmm(a.view(-1), b.view(-1), c, up(indptr), up(cols), nb, mb, nnzb, blk, feat)
    bound = mag * (max(counts) * blk / 16 + 8) * 2.0 ** -23  # as above
    assert bool(((c.view(nb, blk, feat).double() - want).abs() <= bound).all())
