"""SDDMM on short, long and empty rows, with every vector width and alignment, against float64 dot
products."""
import numpy as np
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu

SHAPES = {
    "one_position": [0, 0, 1],
    "singles": [1] * 5001,
    "empty_runs": ([0] * 400 + [1, 2, 3] + [0] * 33 + [5]) * 20,
    "hubs_among_short_rows": [3, 0, 1, 900, 2, 2, 31, 32, 33, 0, 1] * 30,
    "long_rows": [700, 0, 1500, 64, 65],
    # 159,000 positions: groups of 32-byte lanes take five blocks per SM
    "one_round_of_five_blocks": [3, 0, 1, 9, 2, 31, 0, 7] * 3000,
}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("feat,offset", [(1, 0), (8, 0), (23, 0), (31, 0), (33, 0), (46, 0), (56, 0), (64, 0), (100, 0),
                                         (130, 0), (264, 0), (299, 0), (512, 0), (64, 1), (64, 2), (96, 4)])
@pytest.mark.parametrize("scaled", [False, True])
def test_rows_and_alignments(cuda_device, shape, feat, offset, scaled):
    deg = np.asarray(SHAPES[shape], np.int64)
    m, n, nnz = len(deg), 777, int(deg.sum())
    rng = np.random.default_rng(feat)
    dev = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    indptr = np.zeros(m + 1, np.int32)
    indptr[1:] = np.cumsum(deg)
    cols = dev(rng.integers(0, n, nnz).astype(np.int32))
    a = dev(rng.uniform(-1, 1, m * feat + offset).astype(np.float32))[offset:]
    b = dev(rng.uniform(-1, 1, n * feat + offset).astype(np.float32))[offset:]
    scale = dev(rng.uniform(0, 1, nnz).astype(np.float32))
    out = torch.full((nnz,), float("nan"), device=cuda_device)
    ops.sddmm(a, b, out, dev(indptr), cols, *([scale] if scaled else []))
    rows = torch.repeat_interleave(torch.arange(m, device=cuda_device), dev(deg))
    prod = a.view(m, feat)[rows].double() * b.view(n, feat)[cols.long()].double()
    s = scale.double() if scaled else 1.0
    want, mag = prod.sum(1) * s, prod.abs().sum(1) * s
    # an fp32 sum of feat products in any order and one more product: feat + 1 half-ulps of the magnitudes
    assert bool(((out.double() - want).abs() <= mag * (feat + 2) * 2.0 ** -24).all())


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("feat,offset", [(96, 0), (128, 0), (160, 0), (192, 0), (256, 0), (128, 8), (160, 8), (64, 8)])
def test_groups_of_eight_lanes(cuda_device, shape, feat, offset):
    """Whole and partly filled tiles of 64 features, rows on both sides of where the kernels change hands."""
    test_rows_and_alignments(cuda_device, shape, feat, offset, True)


@pytest.mark.parametrize("n,feat,per_row", [(300_000, 64, 100), (150_000, 96, 20), (80_000, 256, 20), (40_000, 512, 20)])
def test_operands_beyond_l2_are_taken_in_slices(cuda_device, n, feat, per_row):
    """Where the rows of B do not stay in L2 as a whole, a call is a launch per slice of them.  It shows in the
    rounding: the products of the first slice sum to 1 and those of a later one to half an ulp of it in 4 lanes' parts, which are
    added up before they meet the 1; a kernel that walks whole rows adds them to the 1 part by part, and loses them."""
    rows = 300
    tile = 32
    while tile < 256 and feat % (2 * tile) == 0 and n * 2 * tile * 4 <= 48 << 20:
        tile *= 2
    assert tile < feat
    b = torch.zeros(n, feat, device=cuda_device)
    b[:, 0] = 1.0
    parts = tile // 8  # 8 features to a lane
    b[:, tile:2 * tile:8] = 2.0 ** -23 / parts
    a = torch.ones(rows * feat, device=cuda_device)
    ptr = torch.arange(0, rows * per_row + 1, per_row, dtype=torch.int32, device=cuda_device)
    cols = torch.randint(0, n, (rows * per_row,), device=cuda_device, dtype=torch.int32)
    out = torch.empty(rows * per_row, device=cuda_device)
    ops.sddmm(a, b.view(-1), out, ptr, cols)
    assert bool((out == 1.0 + 2.0 ** -23).all())


@pytest.mark.parametrize("feat", [8, 24, 40, 56, 64, 72, 120, 128, 136, 192, 200, 248, 264])
@pytest.mark.parametrize("per_row", [9, 10, 16, 33, 64, 200])
def test_tiles_that_rows_do_not_fill(cuda_device, feat, per_row):
    # around the row lengths at which the kernels change, with a row of infinities in B
    m, n = 3001, 801
    g = torch.Generator(device=cuda_device).manual_seed(feat)
    deg = torch.full((m,), per_row, device=cuda_device)
    deg[::7] = 0
    deg[1::7] = 2 * per_row
    ptr = torch.zeros(m + 1, dtype=torch.int32, device=cuda_device)
    ptr[1:] = deg.cumsum(0)
    nnz = int(ptr[-1])
    cols = torch.randint(0, n, (nnz,), generator=g, device=cuda_device, dtype=torch.int32)
    a, b = (torch.rand(k, feat, generator=g, device=cuda_device) - 0.5 for k in (m, n))
    b[5] = float("inf")
    a[:, 0] = 1.0
    a[:, 1:4] = 0.25  # sums of infinities of one sign where only the first piece counts
    a[:, 4:] = a[:, 4:].abs()
    out = torch.full((nnz,), 7.0, device=cuda_device)
    ops.sddmm(a.view(-1), b.view(-1), out, ptr, cols)
    rows = torch.repeat_interleave(torch.arange(m, device=cuda_device), deg)
    prod = a[rows].double() * b[cols.long()].double()
    want, mag = prod.sum(1), prod.abs().sum(1)
    inf = cols == 5
    assert bool((out[inf] == float("inf")).all())
    assert bool(((out.double() - want).abs() <= mag * (feat + 8) * 2.0 ** -24)[~inf].all())


@pytest.mark.parametrize("feat", [24, 40, 64, 104])
@pytest.mark.parametrize("tail", [0, 40])
def test_rows_that_end_inside_a_batch(cuda_device, feat, tail):
    """Batches of 32 positions in which no row, one to six rows and more than 32 rows end, rows without positions among and
    behind them, and a last batch of every length; rows are long enough on average for the kernel that keeps the row of A."""
    rng = np.random.default_rng(feat)
    ends = [[32], [31, 1], [5, 27], [8] * 4, [7, 6, 6, 6, 7], [6, 5, 5, 5, 5, 6], [1] * 32, [0, 0, 32], [16] + [0] * 40 + [16], [3] * 10 + [2]]
    deg = np.array(sum((ends[i] for i in rng.integers(0, len(ends), 900)), []) + [500] * (1800 if feat == 64 else 450) + [13] + [0] * tail)
    deg = np.concatenate([deg[rng.permutation(len(deg) - tail)], deg[len(deg) - tail:]])
    m, nnz, n = len(deg), int(deg.sum()), 4001
    assert nnz >= 120_000 and nnz // m >= (64 if feat == 64 else 24)
    ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).to(cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(feat)
    cols = torch.randint(0, n, (nnz,), generator=g, device=cuda_device, dtype=torch.int32)
    a, b = (torch.rand(k, feat, generator=g, device=cuda_device) - 0.5 for k in (m, n))
    out = torch.full((nnz,), 7.0, device=cuda_device)
    ops.sddmm(a.view(-1), b.view(-1), out, ptr, cols)
    rows = torch.repeat_interleave(torch.arange(m, device=cuda_device), torch.from_numpy(deg).to(cuda_device))
    prod = a[rows].double() * b[cols.long()].double()
    assert bool(((out.double() - prod.sum(1)).abs() <= prod.abs().sum(1) * (feat + 2) * 2.0 ** -24).all())
