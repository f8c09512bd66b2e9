"""fp16 RGMS on buckets of which one has one column per row and many rows: those rows are transformed straight from X
and the others through Z, in launches that overlap.  Whole numbers and halves, so that every order of addition is exact."""
import ctypes

import pytest
import torch

from sparsetir_b200 import _lib as L
from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu

SINGLE = 96 << 10  # rows from which the one-column bucket gets launches of its own


def _layer(device, widths, rows, group, rels, n, m, fi, fo, seed, top=2):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    pick = lambda lo, hi, *shape: torch.randint(lo, hi, shape, device=device, generator=g)  # noqa: E731
    buckets = []
    for width, count in zip(widths, rows):
        groups = -(-count // group)
        vals = (pick(0, 4, groups * group, width).float() / 2).half()  # zeros among them
        mid = torch.sort(pick(0, rels, groups))[0].int()
        buckets.append((vals.view(-1), pick(0, m, groups * group).int(), pick(0, n, groups * group * width).int(), mid))
    x = pick(-top, top + 1, n, fi).half()
    w = pick(-top, top + 1, rels, fi, fo).half()
    want = torch.zeros(m, fo, dtype=torch.float64, device=device)
    for width, (vals, to, cols, mid) in zip(widths, buckets):
        z = (vals.view(-1, width, 1).double() * x[cols.long()].view(-1, width, fi).double()).sum(1)
        rel = torch.repeat_interleave(mid.long(), group)
        for r in range(rels):
            at = torch.nonzero(rel == r)[:, 0]
            want.index_add_(0, to[at].long(), z[at] @ w[r].double())
    return buckets, x, w, want


@pytest.mark.parametrize("widths,rows,group", [((1, 2), (SINGLE, 500), 32), ((4, 1, 2), (1000, SINGLE + 37, 3000), 1),
                                               ((1, 8, 1), (SINGLE + 5000, 300, 2000), 64), ((2, 1), (20_000, SINGLE - 64), 64),
                                               ((1, 1), (SINGLE, SINGLE + 128), 128)])
@pytest.mark.parametrize("fi,fo", [(64, 64), (128, 64), (64, 192), (64, 32)])
def test_exact_sums(cuda_device, widths, rows, group, fi, fo):
    n, m, rels = 700, 4000, 7
    buckets, x, w, want = _layer(cuda_device, widths, rows, group, rels, n, m, fi, fo, len(widths) + fi + fo)
    y = torch.full((m, fo), 2.0, device=cuda_device)
    args = ops.rgms_ell3d_f16_args(w.view(-1), x.view(-1), y.view(-1), buckets, fi, fo)
    ops.rgms_ell3d_f16(*args)
    assert torch.equal(y.double(), want + 2.0)
    count = ctypes.c_uint(0)
    assert L.load().sparsetir_tc_timeouts(cuda_device.index or 0, ctypes.byref(count)) == 0 and count.value == 0


@pytest.mark.parametrize("widths,rows,group", [((1, 2), (SINGLE, 500), 32), ((4, 1, 2), (1000, SINGLE + 37, 3000), 1), ((1, 1), (SINGLE, SINGLE + 128), 128),
                                               ((8, 1, 4), (47_500, SINGLE + 1, 500), 1)])  # at 128 features two tiles of the gather per block
@pytest.mark.parametrize("fi,fo", [(64, 64), (128, 64), (64, 192), (64, 32)])
def test_exact_sums_in_float16(cuda_device, widths, rows, group, fi, fo):
    """The result in half precision: multiples of a half below 1024, which every order of addition keeps."""
    n, m, rels = 700, 40_000, 7
    buckets, x, w, want = _layer(cuda_device, widths, rows, group, rels, n, m, fi, fo, len(widths) + fi + fo, top=1)
    assert float(want.abs().max()) < 500
    y = torch.full((m, fo), 2.0, device=cuda_device, dtype=torch.float16)
    ops.rgms_ell3d_f16(*ops.rgms_ell3d_f16_args(w.view(-1), x.view(-1), y.view(-1), buckets, fi, fo))
    assert torch.equal(y.double(), want + 2.0)


def test_calls_in_a_row_and_in_a_graph(cuda_device):
    """Layers that feed one another without a synchronisation: the overlapping launches of one call are over before the
    next reads the result or overwrites the scratch."""
    n, rels, f = 6000, 7, 64
    buckets, x, w, want = _layer(cuda_device, (1, 2, 4), (SINGLE, 9000, 4000), 4, rels, n, n, f, f, 3)
    y = torch.zeros(n, f, device=cuda_device)
    call = ops.rgms_ell3d_f16.prepare(*ops.rgms_ell3d_f16_args(w.view(-1), x.view(-1), y.view(-1), buckets, f, f))
    x0 = x.clone()
    for _ in range(30):
        y.zero_()
        call()
        assert torch.equal(y.double(), want)
        x.copy_(x0 * 2)  # right behind the call that reads x
        y.zero_()
        call()
        x.copy_(x0)
        assert torch.equal(y.double(), 2 * want)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    assert L.load().sparsetir_reserve_workspace(0, ctypes.c_void_p(stream.cuda_stream), 64 << 20, 1 << 20) == 0
    with torch.cuda.graph(graph, stream=stream):
        y.zero_()
        call()
    for _ in range(10):
        graph.replay()
        assert torch.equal(y.double(), want)
