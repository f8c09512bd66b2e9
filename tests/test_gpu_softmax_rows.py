"""Softmax of a large matrix, whose rows are taken by blocks: row lengths at which a warp's and a block's registers end,
blocks that mix them with short and empty rows, values at the ends of the type, and the result in place of the scores."""
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu

SPECIAL = [511, 512, 513, 0, 1, 31, 32, 33, 4095, 4096, 4097, 8191, 8193, 10_000, 0, 0, 300_000, 127, 128, 129, 2047, 2049]


def _matrix(device, seed):
    """The special rows, among rows that bring the matrix to the size from which blocks take its rows."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    deg = torch.randint(0, 2000, (12_900,), device=device, generator=g)
    deg[torch.randperm(12_900, device=device, generator=g)[:len(SPECIAL)]] = torch.tensor(SPECIAL, device=device)
    ptr = torch.zeros(len(deg) + 1, dtype=torch.int64, device=device)
    ptr[1:] = torch.cumsum(deg, 0)
    assert int(ptr[-1]) >= 12 << 20
    return g, ptr, torch.repeat_interleave(torch.arange(len(deg), device=device), deg)


def _want(a, rows, n):
    a = a.double()
    top = torch.full((n,), -torch.finfo(torch.float32).max, dtype=torch.float64, device=a.device)
    top = top.scatter_reduce(0, rows, a, "amax")
    e = torch.exp(a - top[rows])
    total = torch.zeros(n, dtype=torch.float64, device=a.device).index_add_(0, rows, e)
    return e * (torch.exp(top) / total)[rows]


def test_rows_of_every_length_and_in_place(cuda_device):
    g, ptr, rows = _matrix(cuda_device, 1)
    a = torch.rand(len(rows), device=cuda_device, generator=g) * 12 - 6
    want = _want(a, rows, len(ptr) - 1)
    cols = torch.zeros(len(rows), dtype=torch.int32, device=cuda_device)
    got = torch.full_like(a, 7.0)
    ops.sparse_softmax(a, got, ptr.int(), cols)
    # a - max is below 12 and rounded by 2^-21 at most, an exponential by 2^-22, the sums of up to 1200 values per thread
    # by 2^-24 of the partial sum each, which is 2^-14 at worst for the row of 300,000 and less than 2^-18 for the others
    err = (got.double() - want).abs() / want
    long_row = torch.bincount(rows).argmax()
    assert float(err[rows != long_row].max()) < 2.0 ** -18 and float(err.max()) < 2.0 ** -14
    ops.sparse_softmax(a, a, ptr.int(), cols)
    assert torch.equal(a, got)


def test_rows_of_lowest_values_and_infinities(cuda_device):
    g, ptr, rows = _matrix(cuda_device, 2)
    n = len(ptr) - 1
    a = torch.rand(len(rows), device=cuda_device, generator=g)
    kind = torch.randint(0, 8, (n,), device=cuda_device, generator=g)[rows]
    first = torch.arange(len(rows), device=cuda_device) == ptr[:-1][rows]
    inf = float("inf")
    a[kind == 0] = -inf                      # 0 / 0
    a[(kind == 1) & first] = inf             # inf - inf
    a[(kind == 2) & ~first] = -inf           # one value and nothing beside it
    a[kind == 3] = -3.0e38                   # exp of the maximum is 0
    a[(kind == 4) & first] = float("nan")
    got = torch.empty_like(a)
    cols = torch.zeros(len(rows), dtype=torch.int32, device=cuda_device)
    ops.sparse_softmax(a, got, ptr.int(), cols)
    bad = (kind == 0) | (kind == 1) | (kind == 4)
    assert bool(torch.isnan(got[bad]).all())
    assert bool((got[kind == 3] == 0.0).all())
    torch.testing.assert_close(got[~bad].double(), _want(torch.where(bad, 0.0, a), rows, n)[~bad], rtol=2.0 ** -14, atol=0.0)
    # a row of one value is its exponential
    one = (kind == 2) & first
    torch.testing.assert_close(got[one], torch.exp(a[one]), rtol=2.0 ** -20, atol=0.0)


def test_attention_with_the_scores_in_place(cuda_device):
    g, ptr, rows = _matrix(cuda_device, 3)
    n, f = len(ptr) - 1, 32
    cols = torch.randint(0, n, (len(rows),), device=cuda_device, generator=g, dtype=torch.int32)
    q, k, v = (torch.rand(n * f, device=cuda_device, generator=g) / 4 for _ in range(3))
    o = torch.empty(n * f, device=cuda_device)
    ops.fusedmm(q, k, v, o, ptr.int(), cols)
    s, p, want = torch.empty(len(rows), device=cuda_device), torch.empty(len(rows), device=cuda_device), torch.empty_like(o)
    ops.sddmm(q, k, s, ptr.int(), cols, torch.ones_like(s))
    ops.sparse_softmax(s, p, ptr.int(), cols)
    ops.csrmm(p, v, want, ptr.int(), cols)
    assert torch.equal(o, want)


@pytest.mark.parametrize("length", [600, 1000, 2000])
def test_rows_of_some_hundred_entries_are_not_shared(cuda_device, length):
    """Rows that a warp takes in a few steps: shared by a block, a matrix of them took twice as long.  It shows in the
    rounding: behind the row's largest value, whose exponential is 1, a thread adds values of just less than half an ulp of 1,
    and loses them; a thread of a warp has eight times as many of the row's values as one of a block."""
    n = (12 << 20) // length + 1
    ptr = torch.arange(0, (n + 1) * length, length, dtype=torch.int32, device=cuda_device)
    small = -16.66  # exp: 0.98 * 2^-24
    a = torch.full((n, length), small, device=cuda_device)
    a[:, 0] = 0.0
    got = torch.empty(n * length, device=cuda_device)
    ops.sparse_softmax(a.view(-1), got, ptr, torch.zeros(n * length, dtype=torch.int32, device=cuda_device))
    lost = -(-length // 32) - 1  # the others of the first thread
    term = torch.exp(torch.tensor(small, dtype=torch.float32).double())
    want = 1.0 / (1.0 + (length - 1 - lost) * term)
    # the other sums and the division round by 2^-24 of 1 a few times; of a block's threads the first would lose an
    # eighth of this, and the result be lower by the rest, 0.8 * lost * 2^-24 and more
    assert float((got.view(n, length)[:, 0].double() - want).abs().max()) < 0.3 * lost * 2.0 ** -24
