"""The condensed SpMM with row tiles of every length: empty runs, tiles at the border between one warp and a
window, hub tiles over several windows, feature counts that are not whole slabs."""
import ctypes

import numpy as np
import pytest
import torch

from sparsetir_b200 import _lib as L
from sparsetir_b200 import format as fmt
from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


def matrix(n, rows, seed):
    """CSR of an n x n matrix whose row r has rows[r] random distinct columns, the others none."""
    rng = np.random.default_rng(seed)
    deg = np.zeros(n, np.int64)
    cols = []
    for r, d in sorted(rows.items()):
        deg[r] = d
        cols.append(np.sort(rng.choice(n, d, replace=False)))
    return np.concatenate([[0], np.cumsum(deg)]).astype(np.int32), np.concatenate(cols).astype(np.int32)


MATRICES = {
    "one": (40, {0: 1}),
    "borders": (5000, {0: 256, 16: 257, 40: 272, 64: 255, 100: 4096, 2999: 1}),  # 16 and 17 groups; two windows
    "hubs": (9000, {8: 9000, 4000: 2048, 4016: 2047, 4040: 2049, 8999: 8999}),
    "gaps": (60000, {3: 20, 31000: 3000, 59990: 700, 59999: 16}),  # thousands of empty tiles between
    "dense": (700, {r: 60 + r % 200 for r in range(700)}),
}


@pytest.mark.parametrize("name", sorted(MATRICES))
@pytest.mark.parametrize("t", [8, 16, 32])
@pytest.mark.parametrize("feat", [8, 64, 72, 160])
def test_matches_a_float64_product(cuda_device, name, t, feat):
    n, rows = MATRICES[name]
    indptr, indices = matrix(n, rows, len(name) + t)
    gp, tiles, mask = fmt.condense(indptr, indices, t, 16)
    rng = np.random.default_rng(feat)
    vals = rng.uniform(0.5, 1.5, mask.shape).astype(np.float16) * mask.astype(np.float16)
    mb, nb = len(gp) - 1, -(-n // 16)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).to(cuda_device)  # noqa: E731
    a, gp_d, ids = up(vals), up(gp), up(tiles)
    b = torch.from_numpy(rng.uniform(-1, 1, (nb * 16, feat)).astype(np.float16)).to(cuda_device)
    # the same sums in float64: (group, row, slot) entries that are not zero
    at = torch.nonzero(a)[:, 0]
    group = at // (t * 16)
    row = torch.searchsorted(gp_d.long(), group, right=True) - 1
    row = row * t + at // 16 % t
    col = ids.long()[group * 16 + at % 16]
    want = torch.zeros(mb * t, feat, dtype=torch.float64, device=cuda_device)
    mag, terms = torch.zeros_like(want), torch.zeros(mb * t, dtype=torch.float64, device=cuda_device)
    prod = a[at].double()[:, None] * b[col].double()
    want.index_add_(0, row, prod)
    mag.index_add_(0, row, prod.abs())
    terms.index_add_(0, row, torch.ones_like(row, dtype=torch.float64))
    bound = mag * (terms[:, None] + 4) * 2.0 ** -23  # fp32 sums of exact products, in any order
    for dtype in (torch.float32, torch.float16):
        outs = []
        for _ in range(2):
            c = torch.full((mb * t * feat,), 3.0, dtype=dtype, device=cuda_device)
            ops.tcspmm(a, b.view(-1), c, gp_d, ids, mb, nb, len(tiles), feat, t, 16)
            outs.append(c)
        assert torch.equal(outs[0], outs[1])
        slack = bound if dtype == torch.float32 else bound + want.abs() * 2.0 ** -10 + 2.0 ** -24
        assert bool(((outs[0].view(mb * t, feat).double() - want).abs() <= slack).all())


@pytest.mark.parametrize("feat", [64, 128])
def test_values_that_are_not_finite_reach_their_own_rows_only(cuda_device, feat):
    indptr, indices = matrix(640, {0: 3, 1: 300, 5: 640, 200: 2}, 1)
    gp, tiles, mask = fmt.condense(indptr, indices, 16, 16)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).to(cuda_device)  # noqa: E731
    b = torch.ones(640, feat, dtype=torch.float16, device=cuda_device)
    hit = int(indices[indptr[1]])
    b[hit, 2] = float("inf")
    c = torch.empty(640 * feat, device=cuda_device)
    ops.tcspmm(up(mask).half(), b.view(-1), c, up(gp), up(tiles), 40, 40, len(tiles), feat, 16, 16)
    want = torch.from_numpy(np.diff(indptr).astype(np.float32)).to(cuda_device)[:, None].repeat(1, feat)
    for r in range(640):
        if hit in indices[indptr[r]:indptr[r + 1]]:
            want[r, 2] = float("inf")
    assert torch.equal(c.view(640, feat), want)


def test_unaligned_operands(cuda_device):
    indptr, indices = matrix(500, {r: 7 for r in range(0, 500, 3)}, 2)
    gp, tiles, mask = fmt.condense(indptr, indices, 16, 16)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).to(cuda_device)  # noqa: E731
    b = torch.rand(512 * 72, device=cuda_device).half()
    outs = []
    for shift in (0, 1):
        ids = torch.empty(tiles.size + 1, dtype=torch.int32, device=cuda_device)[shift:][:tiles.size]
        ids.copy_(up(tiles))
        c = torch.empty(32 * 16 * 72 + 1, device=cuda_device)[shift:][:32 * 16 * 72]
        ops.tcspmm(up(mask).half(), b, c, up(gp), ids, 32, 32, len(tiles), 72, 16, 16)
        outs.append(c.clone())
    assert torch.equal(outs[0], outs[1])


def test_long_windows_of_large_products(cuda_device):
    # 4,096 features: windows of 128 groups would need more scratch than the operator takes
    feat, t, n = 4096, 16, 6400
    lengths = [400, 0, 3, 130, 399, 16, 17] + [350] * 60  # groups per row tile
    gp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    groups = int(gp[-1])
    need = [ctypes.c_size_t(0) for _ in range(2)]
    assert L.load().sparsetir_tcspmm_workspace(groups, feat, t, 16, *(ctypes.byref(x) for x in need)) == 0
    assert need[0].value < groups * (feat // 64) * 64  # what windows of 128 groups need: the case is beyond the limit
    rng = np.random.default_rng(0)
    ids = np.concatenate([np.sort(rng.choice(n, g * 16, replace=False)) for g in lengths]).astype(np.int32)
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(cuda_device)  # noqa: E731
    a = torch.rand(groups * t * 16, device=cuda_device).half()
    b = torch.rand(n, feat, device=cuda_device).half()
    c = torch.full((len(lengths) * t * feat,), 3.0, device=cuda_device)
    for _ in range(2):
        ops.tcspmm(a, b.view(-1), c, up(gp), up(ids), len(lengths), n // 16, groups, feat, t, 16)
    for io, g in enumerate(lengths):
        block = a.view(groups, t, 16)[gp[io]:gp[io + 1]].permute(1, 0, 2).reshape(t, -1).double()
        want = block @ b[up(ids[gp[io] * 16:gp[io + 1] * 16]).long()].double()
        # fp32 sums of exact products that are not negative
        assert bool(((c.view(-1, t, feat)[io].double() - want).abs() <= want * (g * 16 + 4) * 2.0 ** -23).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("feat,shift", [(64, 8), (96, 8), (80, 0), (24, 0), (64, 0)])
def test_outputs_with_and_without_whole_sectors(cuda_device, dtype, feat, shift):
    """Results of 32-byte sectors are stored in one piece, others (a result 16 bytes off, rows of 48 bytes) in two."""
    indptr, indices = matrix(700, {r: 1 + r % 30 for r in range(700)}, feat)
    gp, tiles, mask = fmt.condense(indptr, indices, 16, 16)
    mb = len(gp) - 1
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).to(cuda_device)  # noqa: E731
    a, gp_d, ids = up(mask.astype(np.float16)), up(gp), up(tiles)
    b = (torch.randint(-8, 9, (44 * 16 * feat,), device=cuda_device) / 4).half()  # whole quarters: exact sums in any order
    want = torch.zeros(mb * 16, feat, device=cuda_device)
    rows = torch.repeat_interleave(torch.arange(700, device=cuda_device), torch.from_numpy(np.diff(indptr)).to(cuda_device))
    want.index_add_(0, rows, b.view(-1, feat)[torch.from_numpy(indices).to(cuda_device).long()].float())
    buf = torch.full((mb * 16 * feat + 64,), 3.0, dtype=dtype, device=cuda_device)
    c = buf[shift:shift + mb * 16 * feat]
    ops.tcspmm(a, b, c, gp_d, ids, mb, 44, len(tiles), feat, 16, 16)
    assert torch.equal(c.view(-1, feat).float(), want.to(dtype).float())
    assert bool((buf[:shift] == 3.0).all()) and bool((buf[shift + len(c):] == 3.0).all())
