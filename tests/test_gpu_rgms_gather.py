"""rgms_ell3d_f16 over buckets of every width: the aggregation of several rows per thread, ragged last tiles,
and rows of a few or of very many 16-byte pieces."""
import numpy as np
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths", [[1, 2, 4, 8, 16, 32], [2], [3, 5], [1, 7, 9, 24]])
@pytest.mark.parametrize("feat_in,feat_out", [(64, 64), (8, 24), (72, 64), (128, 128), (2048, 64), (12, 16),
                                              (16, 32), (32, 32), (80, 96), (48, 256), (32, 48)])
@pytest.mark.parametrize("groups", [1, 37])
def test_matches_a_float64_product(cuda_device, widths, feat_in, feat_out, groups):
    rng = np.random.default_rng(sum(widths) + feat_in + groups)
    m, n, rels, rows_per_group = 300, 211, 5, 9
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)  # noqa: E731
    x = up(rng.uniform(-1, 1, (n, feat_in)).astype(np.float16))
    w = up((rng.standard_normal((rels, feat_in, feat_out)) / np.sqrt(feat_in)).astype(np.float16))
    want = torch.zeros(m, feat_out, dtype=torch.float64, device=cuda_device)
    mag, adds = torch.zeros_like(want), torch.zeros(m, dtype=torch.float64, device=cuda_device)
    buckets = []
    for width in widths:
        rows = groups * rows_per_group
        a = up(rng.uniform(0, 1, (rows, width)).astype(np.float16))
        cols, ids = up(rng.integers(0, n, (rows, width))), up(rng.integers(0, m, rows))
        mid = up(np.sort(rng.integers(0, rels, groups)).astype(np.int32))
        rel = mid.long().repeat_interleave(rows_per_group)
        z = (a.double()[:, :, None] * x.double()[cols]).sum(1)
        zmag = (a.double()[:, :, None] * x.double()[cols].abs()).sum(1)
        want.index_add_(0, ids, torch.bmm(z[:, None], w.double()[rel])[:, 0])
        mag.index_add_(0, ids, torch.bmm(zmag[:, None], w.double().abs()[rel])[:, 0])
        adds.index_add_(0, ids, torch.ones_like(ids, dtype=torch.float64))
        buckets.append((a.view(-1), ids.int(), cols.int().view(-1), mid))
    y = torch.zeros(m * feat_out, device=cuda_device)
    ops.rgms_ell3d_f16(*ops.rgms_ell3d_f16_args(w.view(-1), x.view(-1), y, [
        (a.view(groups, rows_per_group, -1), r.view(groups, rows_per_group), c.view(groups, rows_per_group, -1), d)
        for a, r, c, d in buckets], feat_in, feat_out))
    # z is rounded to float16 once (its own magnitude, subnormal steps below 2^-14), the rest is fp32
    bound = mag * (2.0 ** -11 + (feat_in + adds[:, None] + 40) * 2.0 ** -23) + adds[:, None] * feat_in * 2.0 ** -25
    assert bool(((y.view(m, feat_out).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("rels", [511, 512, 513])
def test_more_ranges_than_a_block_keeps(cuda_device, rels):
    # (bucket, relation) ranges of two buckets lie in shared memory up to 1,024 of them; most have no rows
    g = torch.Generator(device=cuda_device).manual_seed(rels)
    m, n, feat, groups, rows_per_group = 200, 150, 64, 90, 7
    x = (torch.rand(n, feat, generator=g, device=cuda_device) - 0.5).half()
    w = (torch.randn(rels, feat, feat, generator=g, device=cuda_device) / 8).half()
    want = torch.zeros(m, feat, dtype=torch.float64, device=cuda_device)
    mag, buckets = torch.zeros_like(want), []
    for width in (2, 4):
        a = torch.rand(groups, rows_per_group, width, generator=g, device=cuda_device).half()
        cols = torch.randint(0, n, (groups, rows_per_group, width), generator=g, device=cuda_device)
        ids = torch.randint(0, m, (groups, rows_per_group), generator=g, device=cuda_device)
        mid = torch.randint(0, rels, (groups,), generator=g, device=cuda_device).sort()[0]
        z = (a.double()[..., None] * x.double()[cols]).sum(2)
        zmag = (a.double()[..., None] * x.double().abs()[cols]).sum(2)
        want.index_add_(0, ids.view(-1), torch.bmm(z, w.double()[mid]).view(-1, feat))
        mag.index_add_(0, ids.view(-1), torch.bmm(zmag, w.double().abs()[mid]).view(-1, feat))
        buckets.append((a, ids.int(), cols.int(), mid.int()))
    y = torch.zeros(m * feat, device=cuda_device)
    ops.rgms_ell3d_f16(*ops.rgms_ell3d_f16_args(w.view(-1), x.view(-1), y, buckets, feat, feat))
    bound = mag * (2.0 ** -11 + 150 * 2.0 ** -23) + feat * 2.0 ** -21  # as above
    assert bool(((y.view(m, feat).double() - want).abs() <= bound).all())
