"""rgms with 128 and 256 features: aggregation, then the tiled transform, against float64; calls inside a
capture with and without scratch."""
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


def layer(device, n, rels, edges, feat, seed):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    rel = torch.sort(torch.randint(0, rels, (edges,), device=device, generator=g))[0]
    dst = torch.randint(0, n, (edges,), device=device, generator=g)
    src = torch.randint(0, n, (edges,), device=device, generator=g)
    key = torch.sort((rel * n + dst) * n + src)[0]
    pair, deg = torch.unique_consecutive(key // n, return_counts=True)
    ptr_i = torch.searchsorted(pair, torch.arange(rels + 1, device=device) * n).int()
    ptr_j = torch.cat([torch.zeros(1, dtype=torch.long, device=device), torch.cumsum(deg, 0)])
    a = torch.rand(edges, device=device, generator=g)
    w = torch.randn(rels, feat, feat, device=device, generator=g) / feat ** 0.5
    x = torch.rand(n, feat, device=device, generator=g) * 2 - 1
    return a, w, x, ptr_i, pair, ptr_j, key % n


def product(a, w, x, ptr_i, pair, ptr_j, src):
    n, rel = x.shape[0], pair // x.shape[0]
    row = torch.repeat_interleave(torch.arange(len(pair), device=x.device), ptr_j[1:] - ptr_j[:-1])
    z = torch.zeros(len(pair), x.shape[1], dtype=x.dtype, device=x.device)
    z.index_add_(0, row, a[:, None] * x[src])
    out = torch.zeros(n, x.shape[1], dtype=x.dtype, device=x.device)
    for r in range(w.shape[0]):
        m = rel == r
        out.index_add_(0, pair[m] % n, z[m] @ w[r].T)
    return out


def arguments(a, w, x, ptr_i, pair, ptr_j, src, y):
    return a, w.reshape(-1), x.reshape(-1), y.view(-1), ptr_i, (pair % x.shape[0]).int(), ptr_j.int(), src.int()


@pytest.mark.parametrize("feat", [128, 256])
@pytest.mark.parametrize("n,rels,edges", [(3, 2, 1), (130, 3, 900), (128, 1, 20_000), (4000, 60, 30_000)])
def test_matches_a_float64_product(cuda_device, feat, n, rels, edges):
    args = layer(cuda_device, n, rels, edges, feat, n)
    d = [t.double() if t.is_floating_point() else t for t in args]
    want = product(*d)
    mag = product(d[0], d[1].abs(), d[2].abs(), *d[3:])
    y = torch.full((n, feat), 2.0, device=cuda_device)
    ops.rgms(*arguments(*args, y))
    # fp32 sums: an aggregated row, the transform, the rows of one output on top of its old value
    steps = int((args[5][1:] - args[5][:-1]).max()) + feat + rels + 1
    assert bool(((y.double() - 2.0 - want).abs() <= (mag + 2.0) * steps * 2.0 ** -24).all())


@pytest.mark.parametrize("warm", [False, True])
def test_inside_a_capture(cuda_device, warm):
    args = layer(cuda_device, 500, 5, 4000, 128, 3)
    want, y = torch.zeros(500, 128, device=cuda_device), torch.zeros(500, 128, device=cuda_device)
    ops.rgms(*arguments(*args, want))
    call = arguments(*args, y)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    if warm:
        with torch.cuda.stream(stream):
            ops.rgms(*call)
        stream.synchronize()
        y.zero_()
        torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        ops.rgms(*call)
    graph.replay()
    torch.cuda.synchronize()
    torch.testing.assert_close(y, want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("feat", [128, 256])
def test_rows_that_a_block_shares(cuda_device, feat):
    """(relation, destination) pairs of 63 to 66 edges and of thousands, beside rows of one and two edges and of none."""
    lens = torch.tensor(([1, 2, 0, 1, 63, 1, 64, 0, 65, 66] + [1, 0, 2] * 40) * 6 + [3000, 0, 700], device=cuda_device)
    n, rels, pairs = 1500, 2, len(lens)
    g = torch.Generator(device=cuda_device).manual_seed(feat)
    ptr_j = torch.cat([torch.zeros(1, dtype=torch.long, device=cuda_device), lens.cumsum(0)])
    edges = int(ptr_j[-1])
    ptr_i = torch.tensor([0, 500, pairs], device=cuda_device).int()
    at = torch.arange(pairs, device=cuda_device)
    pair = at + (at >= 500) * (n - 500)  # rows 0, 1, ... of each relation
    a, x = torch.rand(edges, device=cuda_device, generator=g), torch.rand(n, feat, device=cuda_device, generator=g) * 2 - 1
    w = torch.randn(rels, feat, feat, device=cuda_device, generator=g) / feat ** 0.5
    src = torch.randint(0, n, (edges,), device=cuda_device, generator=g)
    args = a, w, x, ptr_i, pair, ptr_j, src
    d = [t.double() if t.is_floating_point() else t for t in args]
    want, mag = product(*d), product(d[0], d[1].abs(), d[2].abs(), *d[3:])
    y = torch.full((n, feat), 2.0, device=cuda_device)
    ops.rgms(*arguments(*args, y))
    assert bool(((y.double() - 2.0 - want).abs() <= (mag + 2.0) * (int(lens.max()) + feat + rels + 1) * 2.0 ** -24).all())
