"""CSR SpMM split by stored entries: rows that cross sub-warps, blocks and feature tiles, runs of
rows without entries, and every vector width, against a float64 product."""
import numpy as np
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu

# degree sequences; all but the first have 8,192 rows or 65,536 entries, where the split begins
SHAPES = {
    "hubs_in_a_small_matrix": [0, 3, 1500, 65, 64, 0, 2, 900] + [5] * 700 + [700],
    # four times the average row is 169: rows up to that stay with their sub-warp
    "hubs_among_long_rows": [40] * 300 + [0, 165, 169, 170, 900, 171] + [40] * 300 + [170],
    "one_row_of_everything": [0] * 40 + [70_001] + [0] * 9000,
    "rows_longer_than_a_block": [9000, 1, 0, 17_000, 2] * 4,
    "empty_runs": ([0] * 5000 + [1] * 40) * 5 + [0] * 3000,
    "single_entries": [1] * 70_003,
    "mixed": [0, 1, 2, 300, 7, 0, 0, 33, 32, 31] * 1700,
    # shares of a sub-warp that are more than one batch of entries and not a whole number of them
    "shares_of_40_entries": [4, 0, 9, 1, 3, 11, 2, 5, 0, 6] * 1000,
    "shares_of_24_to_80_entries": [9, 0, 20, 1, 13, 2, 45, 0] * 1000,
}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("feat,offset", [(32, 0), (64, 0), (100, 0), (300, 0), (41, 0), (46, 0), (299, 0), (130, 0), (1, 0),
                                         (64, 1), (128, 2), (384, 0), (512, 0), (640, 0)])
def test_rows_meet_across_sub_warps_and_blocks(cuda_device, shape, feat, offset):
    deg = np.asarray(SHAPES[shape], np.int64)
    m, n, nnz = len(deg), 4001, int(deg.sum())
    rng = np.random.default_rng(feat)
    indptr = np.zeros(m + 1, np.int32)
    indptr[1:] = np.cumsum(deg)
    dev = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    cols = dev(rng.integers(0, n, nnz).astype(np.int32))
    vals = dev(rng.uniform(-1, 1, nnz).astype(np.float32))
    x = dev(rng.uniform(-1, 1, n * feat + offset).astype(np.float32))[offset:]  # offset: other alignments
    y = torch.full((m * feat + offset,), float("nan"), device=cuda_device)[offset:]
    ptr = dev(indptr)
    ops.csrmm(vals, x, y, ptr, cols)
    rows = torch.repeat_interleave(torch.arange(m, device=cuda_device), dev(deg))
    want = torch.zeros(m, feat, dtype=torch.float64, device=cuda_device)
    mag = torch.zeros(m, feat, dtype=torch.float64, device=cuda_device)
    for p in range(0, nnz, 20_000):
        part = vals[p:p + 20_000, None].double() * x.view(n, feat)[cols[p:p + 20_000].long()].double()
        want.index_add_(0, rows[p:p + 20_000], part)
        mag.index_add_(0, rows[p:p + 20_000], part.abs())
    # an fp32 sum of d products in any order: at most d half-ulps of the sum of magnitudes
    bound = mag * (dev(deg)[:, None].double() + 1) * 2.0 ** -24
    assert bool(((y.view(m, feat).double() - want).abs() <= bound).all())
    again = y.clone()
    ops.csrmm(vals, x, y, ptr, cols)
    assert torch.equal(again, y)  # one writer and one order: the same bits


@pytest.mark.parametrize("feat", [36, 64, 68, 128, 132, 256])
@pytest.mark.parametrize("deg", [[0, 1, 2, 30, 7, 0, 0, 13, 32, 11] * 1100, [3000, 8, 0] * 10 + [8] * 10_000, [99] * 1200, [100] * 1200, [101] * 1200,
                                 [12, 0, 4] * 5000, [12, 0, 4] * 4999 + [12, 0, 3],
                                 [0, 1, 2, 60, 7, 0, 0, 43, 32, 15] * 900, [2000, 11, 0] * 10 + [11] * 8000],
                         ids=["mixed", "hubs", "below", "long", "longer", "least", "less", "mixed_16", "hubs_13"])
def test_two_vectors_per_lane(cuda_device, deg, feat):
    # more and less than 80,000 and 100,000 entries, rows of 5 to 13 on average, and rows of 99, 100 and 101: from 100 on whole tiles (64, 128 and 256 features) go
    # back to one vector
    deg = torch.tensor(deg, device=cuda_device)
    m, n, nnz = len(deg), 2003, int(deg.sum())
    g = torch.Generator(device=cuda_device).manual_seed(feat)
    ptr = torch.zeros(m + 1, dtype=torch.int32, device=cuda_device)
    ptr[1:] = deg.cumsum(0)
    cols = torch.randint(0, n, (nnz,), generator=g, device=cuda_device, dtype=torch.int32)
    vals = torch.rand(nnz, generator=g, device=cuda_device) - 0.5
    x = torch.rand(n, feat, generator=g, device=cuda_device) - 0.5
    y = torch.full((m * feat,), float("nan"), device=cuda_device)
    ops.csrmm(vals, x.view(-1), y, ptr, cols)
    a = torch.sparse_csr_tensor(ptr, cols, vals.double(), (m, n))
    mag = torch.sparse_csr_tensor(ptr, cols, vals.abs().double(), (m, n)) @ x.abs().double()
    # a sum of d fp32 products in any order: at most d half-ulps of the sum of magnitudes
    assert bool(((y.view(m, feat).double() - a @ x.double()).abs() <= mag * (deg[:, None] + 1) * 2.0 ** -24).all())
    again = y.clone()
    ops.csrmm(vals, x.view(-1), y, ptr, cols)
    assert torch.equal(again, y)


def test_a_prime_number_of_feature_tiles(cuda_device):
    # 65,537 tiles of 160 features: more blocks than a grid can have if every tile had its own
    feat, n, deg = 65_537 * 160 - 1, 2, [2, 0, 1]
    g = torch.Generator(device=cuda_device).manual_seed(1)
    ptr = torch.tensor([0, 2, 2, 3], dtype=torch.int32, device=cuda_device)
    cols = torch.tensor([1, 0, 1], dtype=torch.int32, device=cuda_device)
    vals = torch.rand(3, generator=g, device=cuda_device) - 0.5
    x = torch.rand(n, feat, generator=g, device=cuda_device) - 0.5
    y = torch.full((len(deg), feat), float("nan"), device=cuda_device)
    ops.csrmm(vals, x.view(-1), y.view(-1), ptr, cols)
    want = torch.stack([vals[0].double() * x[1] + vals[1].double() * x[0], torch.zeros_like(x[0]).double(), vals[2].double() * x[1]])
    mag = torch.stack([(vals[0] * x[1]).abs() + (vals[1] * x[0]).abs(), torch.zeros_like(x[0]), (vals[2] * x[1]).abs()]).double()
    # two products and their sum, or one product: at most three half-ulps of the sum of magnitudes
    assert bool(((y.double() - want).abs() <= mag * 3 * 2.0 ** -24).all())


def test_first_call_on_a_stream_can_be_captured(cuda_device):
    m, feat = 9000, 41
    ptr = torch.arange(0, 8 * m + 1, 8, dtype=torch.int32, device=cuda_device)
    cols = torch.randint(0, m, (8 * m,), dtype=torch.int32, device=cuda_device)
    vals, x = torch.rand(8 * m, device=cuda_device), torch.rand(m * feat, device=cuda_device)
    want, got = torch.empty(m * feat, device=cuda_device), torch.empty(m * feat, device=cuda_device)
    ops.csrmm(vals, x, want, ptr, cols)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        ops.csrmm(vals, x, got, ptr, cols)
    for _ in range(2):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


@pytest.mark.parametrize("feat", [64, 41, 100, 512])
@pytest.mark.parametrize("front,behind", [(0, 700), (1000, 0), (12_345, 30_000), (40_000, 1)])
def test_entries_outside_the_row_pointers_count_for_nothing(cuda_device, feat, front, behind):
    # row pointers of a row slice that start behind 0, and arrays with room behind the last row
    rng = np.random.default_rng(feat)
    m, n = 9000, 3000
    deg = rng.poisson(7, m)
    deg[[0, 1, 4000, 8998, 8999]] = [0, 3000, 5000, 700, 0]
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    nnz = int(indptr[-1])
    dev = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    cols = dev(rng.integers(0, n, front + nnz + behind).astype(np.int32))
    vals = torch.full((front + nnz + behind,), float("nan"), device=cuda_device)
    vals[front:front + nnz] = torch.rand(nnz, device=cuda_device)
    x = torch.rand(n * feat, device=cuda_device)
    want, got, after = (torch.empty(m * feat, device=cuda_device) for _ in range(3))
    ptr = dev(indptr)
    ops.csrmm(vals[front:front + nnz].clone(), x, want, ptr, cols[front:front + nnz].clone())
    ops.csrmm(vals, x, got, ptr + front, cols)
    # blocks of other entries each: the same sums, the pieces of a row cut elsewhere
    torch.testing.assert_close(got, want, rtol=5000 * 2.0 ** -24, atol=0)  # of up to 5,000 terms that are not negative
    ops.csrmm(vals[front:front + nnz].clone(), x, after, ptr, cols[front:front + nnz].clone())
    assert torch.equal(after, want)  # the call before left the counters at zero
