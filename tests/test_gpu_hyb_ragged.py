"""hyb SpMM on feature counts that are not whole tiles and operands of every alignment, with rows
that are split over several ELL rows, against a float64 product."""
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
    y = torch.zeros(m * feat + offset, device=cuda_device)[offset:]
    flags = L.HYB_ZERO_C | (L.HYB_ALL_ATOMIC if parts > 1 else 0)
    for _ in range(2):
        ops.hyb_spmm(*ops.hyb_args(x, y, bk, feat, flags))
    a = torch.zeros(m, n, dtype=torch.float64, device=cuda_device)
    a[torch.from_numpy(np.repeat(np.arange(m), deg)).to(cuda_device), dev(cols).long()] = dev(vals).double()
    want, mag = a @ x.view(n, feat).double(), a.abs() @ x.view(n, feat).double().abs()
    # an fp32 sum of d products in any order: at most d half-ulps of the sum of magnitudes
    bound = mag * (dev(deg)[:, None].double() + 1) * 2.0 ** -24
    assert bool(((y.view(m, feat).double() - want).abs() <= bound).all())
