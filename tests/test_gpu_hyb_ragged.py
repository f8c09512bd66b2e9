"""hyb SpMM on feature counts that are not whole tiles and operands of every alignment, with rows
that are split over several ELL rows, against a float64 product."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from sparsetir_b200 import _lib as L
from sparsetir_b200 import format as fmt
from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("buckets", [[1, 2, 4, 8, 16, 32, 64], [1, 4, 512], [8, 24]])
@pytest.mark.parametrize("parts", [1, 2])
@pytest.mark.parametrize("feat,offset", [(1, 0), (31, 0), (33, 0), (41, 0), (66, 0), (100, 0), (130, 0), (184, 0), (264, 0),
                                         (299, 0), (64, 1), (128, 2), (36, 4)])
def test_ragged_features_and_alignments(cuda_device, buckets, parts, feat, offset):
    rng = np.random.default_rng(feat)
    n = 3000
    deg = np.concatenate([[2900, 1300, 520, 513, 512, 0], rng.integers(0, 9, 900)]).astype(np.int64)
    m, nnz = len(deg), int(deg.sum())
    indptr = np.zeros(m + 1, np.int32)
    indptr[1:] = np.cumsum(deg)
    cols = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in deg]).astype(np.int32)
    vals = rng.uniform(-1, 1, nnz).astype(np.float32)
    r, c, _, v, _ = fmt.column_part_hyb(m, n, indptr, cols, parts, buckets, data=vals)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)  # noqa: E731
    bk = [(dev(v[p][b]), dev(r[p][b]), dev(c[p][b])) for p in range(parts) for b in range(len(buckets)) if len(r[p][b])]
    x = dev(rng.uniform(-1, 1, n * feat + offset).astype(np.float32))[offset:]
    named = dev((deg > 0)[:, None].repeat(feat, 1).reshape(-1))
    flags = L.HYB_ALL_ATOMIC | L.HYB_ZERO_C if parts > 1 else 0
    y = torch.zeros(m * feat + offset, device=cuda_device)[offset:]
    if parts == 1:  # no row needs clearing, and rows that occur in no bucket stay as they are
        y[named] = float("nan")
    for _ in range(2):
        ops.hyb_spmm(*ops.hyb_args(x, y, bk, feat, flags))
    a = torch.zeros(m, n, dtype=torch.float64, device=cuda_device)
    a[torch.from_numpy(np.repeat(np.arange(m), deg)).to(cuda_device), dev(cols).long()] = dev(vals).double()
    want, mag = a @ x.view(n, feat).double(), a.abs() @ x.view(n, feat).double().abs()
    # an fp32 sum of d products in any order: at most d half-ulps of the sum of magnitudes
    bound = mag * (dev(deg)[:, None].double() + 1) * 2.0 ** -24
    assert bool(((y.view(m, feat).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("low,high", [(0, 9), (9, 80)])
@pytest.mark.parametrize("parts", [1, 2])
@pytest.mark.parametrize("n,feat", [(3000, 32), (3000, 64), (3000, 100), (3000, 128), (3000, 256), (3000, 260), (110000, 300), (110000, 320)])
def test_ids_by_shuffles_and_through_shared_memory(cuda_device, n, feat, parts, low, high):
    """Short and long rows, on tiles of 8, 16 and 32 lanes (16 where a slice of b is more than L2 keeps), one tile and several, whole and
    partly filled, with rows of 8 slots to rows that a block shares, and partly filled batches in all of them."""
    rng = np.random.default_rng(feat + high)
    deg = np.concatenate([[2900, 1300, 520, 257, 8, 9, 0], rng.integers(low, high, 800)]).astype(np.int64)
    m, nnz, buckets = len(deg), int(deg.sum()), [8, 24, 64, 512]
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in deg]).astype(np.int32)
    vals = rng.uniform(-1, 1, nnz).astype(np.float32)
    if low == 0:
        buckets = [1, 2, 4] + buckets
    r, c, _, v, _ = fmt.column_part_hyb(m, n, indptr, cols, parts, buckets, data=vals)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)  # noqa: E731
    bk = [(dev(v[p][b]), dev(r[p][b]), dev(c[p][b])) for p in range(parts) for b in range(len(buckets)) if len(r[p][b])]
    x = torch.rand(n, feat, generator=torch.Generator(cuda_device).manual_seed(feat), device=cuda_device) * 2 - 1
    y = torch.zeros(m, feat, device=cuda_device)
    for _ in range(2):
        ops.hyb_spmm(*ops.hyb_args(x.view(-1), y.view(-1), bk, feat, L.HYB_ALL_ATOMIC | L.HYB_ZERO_C if parts > 1 else 0))
    a = torch.sparse_csr_tensor(dev(indptr).long(), dev(cols).long(), dev(vals).double(), (m, n))
    want = a @ x.double()
    mag = torch.sparse_csr_tensor(dev(indptr).long(), dev(cols).long(), dev(vals).double().abs(), (m, n)) @ x.double().abs()
    # an fp32 sum of d products in any order: at most d half-ulps of the sum of magnitudes
    assert bool(((y.double() - want).abs() <= mag * (dev(deg)[:, None].double() + 1) * 2.0 ** -24).all())


@pytest.mark.parametrize("feat,lanes,floats", [(512, 32, 4), (64, 8, 4), (130, 32, 2), (256, 32, 4)])
@pytest.mark.parametrize("buckets", [[1, 2, 4, 8], [4, 8, 24]])
def test_items_that_fill_one_wave(cuda_device, feat, lanes, floats, buckets):
    """Calls of a little more than one wave of blocks, whose items are made longer: numbers of rows per item that are no power of two, in
    every bucket, with rows split over items of the widest one."""
    rng = np.random.default_rng(feat)
    n, rows, top = 3000, 60_000, buckets[-1]
    deg = np.minimum(rng.integers(1, 14, rows), top)
    if top == 24:
        deg[::5] = rng.integers(9, 25, rows // 5)
    tiles, per_block = -(-feat // (lanes * floats * (2 if floats == 2 else 1))), 128 // lanes

    def blocks(deg, item=lanes * floats):
        width = np.array(buckets)[np.searchsorted(buckets, np.minimum(deg, top))]
        ell = np.where(deg > top, -(-deg // top), 1)
        return sum(-(-int(ell[width == w].sum()) // (per_block * max(1, item // w))) for w in buckets) * tiles / (8 * 148)

    deg = np.concatenate([[2900, 100, 30, 1300], deg[:next(k for k in range(1000, rows, 250) if blocks(deg[:k]) > 1.03)], [60, 2000]])
    deg = deg[rng.permutation(len(deg))]
    assert 1.0 < blocks(deg) < (1.1 if top == 8 else 1.35)
    m = len(deg)
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    cols = np.concatenate([np.sort((k + np.arange(d) * (n // d)) % n) for k, d in zip(rng.integers(0, n, m), deg)]).astype(np.int32)
    vals = rng.uniform(-1, 1, len(cols)).astype(np.float32)
    r, c, _, v, _ = fmt.column_part_hyb(m, n, indptr, cols, 1, buckets, data=vals)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)  # noqa: E731
    bk = [(dev(v[0][b]), dev(r[0][b]), dev(c[0][b])) for b in range(len(buckets)) if len(r[0][b])]
    x = torch.rand(n, feat, generator=torch.Generator(cuda_device).manual_seed(feat), device=cuda_device) * 2 - 1
    y = torch.full((m, feat), float("nan"), device=cuda_device)
    for _ in range(2):
        ops.hyb_spmm(*ops.hyb_args(x.view(-1), y.view(-1), bk, feat, 0))
    a = torch.sparse_csr_tensor(dev(indptr).long(), dev(cols).long(), dev(vals).double(), (m, n))
    mag = torch.sparse_csr_tensor(dev(indptr).long(), dev(cols).long(), dev(vals).double().abs(), (m, n)) @ x.double().abs()
    assert bool(((y.double() - a @ x.double()).abs() <= mag * (dev(deg)[:, None].double() + 1) * 2.0 ** -24).all())


BEYOND_THE_LIMIT = """
import numpy as np, torch
from sparsetir_b200 import format as fmt, ops
rng = np.random.default_rng(0)
deg = np.concatenate([[2900, 0, 520, 0], rng.integers(0, 9, 900)])
ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
cols = np.concatenate([np.sort(rng.choice(3000, d, replace=False)) for d in deg]).astype(np.int32)
vals = rng.uniform(0.5, 1, len(cols)).astype(np.float32)
r, c, _, v, _ = fmt.column_part_hyb(len(deg), 3000, ptr, cols, 1, [1, 4, 8], data=vals)
up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
buckets = [(up(v[0][b]), up(r[0][b]), up(c[0][b])) for b in range(3)]
a = torch.zeros(len(deg), 3000, dtype=torch.float64, device="cuda")
a[up(np.repeat(np.arange(len(deg)), deg)), up(cols).long()] = up(vals).double()
for feat in (64, 41, 100, 130):
    x, y = torch.rand(3000, feat, device="cuda"), torch.full((len(deg), feat), 3.0, device="cuda")
    for _ in range(2):
        ops.hyb_spmm(*ops.hyb_args(x, y, buckets, feat))
    want = a @ x.double()
    want[up(deg == 0)] = 3.0
    # up to 2,900 terms that are not negative, in any order
    torch.testing.assert_close(y.double(), want, rtol=2901 * 2.0 ** -24, atol=0)
print("done")
"""


def test_without_scratch_rows_of_no_bucket_stay_and_calls_repeat(cuda_device):
    # SPARSETIR_HYB_SCRATCH_MB=0 (read once per process): split rows are added atomically into cleared rows
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", BEYOND_THE_LIMIT], env=dict(os.environ, SPARSETIR_HYB_SCRATCH_MB="0"), cwd=root,
                       capture_output=True, text=True, timeout=600)
    assert (r.returncode, r.stdout.split()) == (0, ["done"]), r.stderr[-2000:]
