"""Calls that follow one another on a stream without a synchronisation: a launch may be scheduled before the one ahead of it
has ended, and must still see all that it wrote (launch.cuh)."""
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


def _graph(n, per_row, device, seed):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    deg = torch.randint(0, 2 * per_row, (n,), device=device, generator=g)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=device)
    ptr[1:] = torch.cumsum(deg, 0)
    nnz = int(ptr[-1])
    cols = torch.randint(0, n, (nnz,), device=device, generator=g, dtype=torch.int32)
    return ptr.int(), cols, torch.rand(nnz, device=device, generator=g) / (8 * per_row)


@pytest.mark.parametrize("n,feat,per_row", [(700, 64, 6), (3000, 32, 3), (20_000, 64, 5), (9000, 100, 20), (3000, 41, 40)])
def test_results_feed_the_next_call(cuda_device, n, feat, per_row):
    """Each call reads what the one before wrote and overwrites what the one before read, fp32 and fp16, with
    torch's own kernels among them: the same bits as with a synchronisation behind every call."""
    ptr, cols, vals = _graph(n, per_row, cuda_device, n)
    x0 = torch.rand(n * feat, device=cuda_device)

    def run(sync):
        x, y = x0.clone(), torch.zeros_like(x0)
        s, p = torch.empty_like(vals), torch.empty_like(vals)
        stop = torch.cuda.synchronize if sync else (lambda: None)
        for _ in range(12):
            ops.csrmm(vals, x, y, ptr, cols); stop()
            ops.sddmm(y, x, s, ptr, cols, vals); stop()
            ops.sparse_softmax(s, p, ptr, cols); stop()
            ops.csrmm(p, y, x, ptr, cols); stop()
            x.mul_(0.01); stop()  # the softmax is not normalised: its results grow with the scores
            ops.fusedmm(x, y, x0, y, ptr, cols); stop()
        torch.cuda.synchronize()
        return x, y, s, p

    want = run(True)
    assert all(bool(torch.isfinite(t).all()) for t in want)
    for _ in range(3):
        for a, b in zip(run(False), want):
            assert torch.equal(a, b)


def test_chain_in_a_graph_and_behind_an_event(cuda_device):
    n, feat = 3000, 64
    ptr, cols, vals = _graph(n, 5, cuda_device, 1)
    x, y, z = (torch.rand(n * feat, device=cuda_device) for _ in range(3))
    calls = [ops.csrmm.prepare(vals, x, y, ptr, cols), ops.csrmm.prepare(vals, y, z, ptr, cols)]
    ops.csrmm(vals, x, y, ptr, cols)
    ops.csrmm(vals, y, z, ptr, cols)
    want = z.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for c in calls:
            c()
    for _ in range(5):
        y.fill_(-1.0), z.fill_(-2.0)
        graph.replay()
        assert torch.equal(z, want)
    # the second call on another stream, held back by an event alone
    side = torch.cuda.Stream()
    for _ in range(20):
        y.fill_(-1.0), z.fill_(-2.0)
        calls[0]()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            calls[1]()
        torch.cuda.current_stream().wait_stream(side)
        assert torch.equal(z, want)


@pytest.mark.parametrize("blk,nb,feat", [(32, 16, 256), (32, 16, 128), (16, 40, 64), (32, 40, 96)])
def test_block_products_feed_the_next_call(cuda_device, blk, nb, feat):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(blk + feat)
    ptr = torch.arange(0, 3 * nb + 1, 3, dtype=torch.int32, device=cuda_device)
    cols = torch.randint(0, nb, (3 * nb,), device=cuda_device, generator=g, dtype=torch.int32)
    a = (torch.rand(3 * nb * blk * blk, device=cuda_device, generator=g) / blk).half()
    b0 = torch.rand(nb * blk * feat, device=cuda_device, generator=g).half()

    def run(sync):
        b, c = b0.clone(), torch.zeros(nb * blk * feat, device=cuda_device)
        for _ in range(20):
            ops.bsrmm(a, b, c, ptr, cols, nb, nb, 3 * nb, blk, feat)
            if sync:
                torch.cuda.synchronize()
            b.copy_(c)
        return c

    want = run(True)
    assert bool(torch.isfinite(want).all())
    for _ in range(3):
        assert torch.equal(run(False), want)
