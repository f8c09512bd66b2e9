"""RGMS at 64 features: rows of one edge, which the transform takes from X, beside rows of none and of many, at the edges of its
tiles and of the groups of the first launch."""
import pytest
import torch

from sparsetir_b200 import _lib as L
from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu
F = 64


def layer(cuda_device, lens, rows_of_relation, n, shift, seed):
    """CSF arrays whose row t has lens[t] entries, X `shift` floats behind a 512-byte boundary, Y of n rows."""
    g = torch.Generator(device=cuda_device).manual_seed(seed)
    lens = torch.tensor(lens, device=cuda_device)
    ptr_j = torch.zeros(len(lens) + 1, dtype=torch.int32, device=cuda_device)
    ptr_j[1:] = lens.cumsum(0)
    ptr_i = torch.tensor([0] + rows_of_relation, device=cuda_device).cumsum(0).int()
    assert int(ptr_i[-1]) == len(lens)
    nnz, rels = int(ptr_j[-1]), len(rows_of_relation)
    rows = torch.cat([torch.randperm(n, generator=g, device=cuda_device)[:k] for k in rows_of_relation]).int()
    cols = torch.randint(0, n, (nnz,), generator=g, device=cuda_device, dtype=torch.int32)
    a = torch.rand(nnz, generator=g, device=cuda_device) + 0.5
    w = torch.randn(rels * F * F, generator=g, device=cuda_device) / 8
    x = (torch.rand(n * F + shift, generator=g, device=cuda_device) - 0.5)[shift:]
    return a, w, x, ptr_i, rows, ptr_j, cols


def exact(a, w, x, ptr_i, rows, ptr_j, cols, n):
    rels, pairs = len(ptr_i) - 1, len(rows)
    rel = torch.repeat_interleave(torch.arange(rels, device=a.device), ptr_i.diff().long())
    row = torch.repeat_interleave(torch.arange(pairs, device=a.device), ptr_j.diff().long())
    x, w = x.view(-1, F).double(), w.view(rels, F, F).double()
    out = []
    for f in (lambda v: v, torch.abs):
        z = torch.zeros(pairs, F, dtype=torch.float64, device=a.device).index_add_(0, row, f(a.double()[:, None] * x[cols.long()]))
        y = torch.zeros(n, F, dtype=torch.float64, device=a.device)
        for r in range(rels):
            at = rel == r
            y.index_add_(0, rows[at].long(), z[at] @ f(w[r]).T)
        out.append(y)
    return out


@pytest.mark.parametrize("lens,relations", [
    ([1], [1]), ([0], [1]), ([0, 1, 2, 0, 3] * 51 + [1], [127, 129]), ([1] * 385, [128, 129, 0, 128]), ([1, 2] * 4097, [8000, 194]),
    ([700, 1, 0, 1, 2, 33] * 40, [239, 1]), ([2, 0, 0, 1, 1, 1, 9, 1] * 10_000, [30_000, 50_000]),
    # rows that all groups of a block share, from 65 entries on, alone and next to each other, in both forms of the first launch
    ([64, 65, 66, 1, 0, 2] + [1, 2] * 400 + [5_000, 300], [807, 1]), (([1, 0, 2, 1, 1, 1, 1, 2] * 99 + [65, 0, 900, 257, 1, 64, 66, 511]) * 50, [40_000])],
    ids=["one", "none", "mixed", "ones", "pairs", "hubs", "many", "shared", "shared_many"])
@pytest.mark.parametrize("shift", [0, 4])
def test_rows_of_one_edge(cuda_device, lens, relations, shift):
    n = 50_000
    a, w, x, ptr_i, rows, ptr_j, cols = layer(cuda_device, lens, relations, n, shift, len(lens))
    y = torch.zeros(n * F, device=cuda_device)
    ops.rgms(a, w, x, y, ptr_i, rows, ptr_j, cols)
    want, mag = exact(a, w, x, ptr_i, rows, ptr_j, cols, n)
    # sums of up to max(lens) + 64 products of three factors, of which the tensor core keeps 21 bits
    bound = mag * ((max(lens) + 64 + 2 * len(relations)) * 2.0 ** -24 + 2.0 ** -20)
    assert bool(((y.view(n, F).double() - want).abs() <= bound).all())
    count = L.ctypes.c_uint(0)
    assert L.load().sparsetir_tc_timeouts(0, L.ctypes.byref(count)) == 0 and count.value == 0


@pytest.mark.parametrize("rels", [1023, 1024, 1025, 3000])
def test_more_relations_than_a_block_keeps(cuda_device, rels):
    # the row ranges lie in shared memory up to 1,024 relations; two of three have no row
    relations = [(r % 3 == 0) * (1 + 130 * (r % 100 == 0)) for r in range(rels)]
    lens = [1, 2, 0, 5] * (sum(relations) // 4 + 1)
    n = 500
    parts = layer(cuda_device, lens[:sum(relations)], relations, n, 0, rels)
    y = torch.zeros(n * F, device=cuda_device)
    ops.rgms(parts[0], parts[1], parts[2], y, *parts[3:])
    want, mag = exact(*parts, n)
    assert bool(((y.view(n, F).double() - want).abs() <= mag * ((5 + 64 + 2 * rels) * 2.0 ** -24 + 2.0 ** -20)).all())


def test_an_infinite_row_reaches_its_destinations_only(cuda_device):
    n, lens = 400, [1, 2, 0, 1] * 75
    a, w, x, ptr_i, rows, ptr_j, cols = layer(cuda_device, lens, [300], n, 0, 3)
    x.view(n, F)[7] = float("inf")
    y = torch.zeros(n * F, device=cuda_device)
    ops.rgms(a, w, x, y, ptr_i, rows, ptr_j, cols)
    row = torch.repeat_interleave(torch.arange(300, device=cuda_device), ptr_j.diff().long())
    hit = torch.zeros(n, dtype=torch.bool, device=cuda_device)
    hit[rows[row[cols == 7]].long()] = True
    assert bool((~torch.isfinite(y.view(n, F))).any(1).eq(hit).all())
