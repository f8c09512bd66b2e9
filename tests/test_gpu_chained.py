"""Calls that follow one another on a stream without a synchronisation: a launch may be scheduled before the one ahead of it
has ended, and must still see all that it wrote (launch.cuh)."""
import numpy as np
import pytest
import torch

from sparsetir_b200 import format as fmt
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


# ---- chains of library calls alone: nothing of torch between a call and the next that reads, or overwrites, its operands

def _same_without_waiting(run, times=3):
    """``run(stop)`` returns what a chain computes; ``stop`` is called behind every call.  The same bits with and without."""
    want = run(torch.cuda.synchronize)
    assert all(bool(torch.isfinite(t).all()) and bool((t != 0).any()) for t in want)
    for _ in range(times):
        for got, ref in zip(run(lambda: None), want):
            assert torch.equal(got, ref)


@pytest.mark.parametrize("blk,nb,feat", [(32, 64, 512), (32, 64, 128), (32, 64, 96), (16, 100, 64), (64, 24, 64)])
def test_block_products_are_gathered_at_once(cuda_device, blk, nb, feat):
    """Every form of the block product, whose result a CSR product reads and the next block product overwrites."""
    n, per = nb * blk, 5
    g = torch.Generator(device=cuda_device)
    g.manual_seed(blk + feat)
    bptr = torch.arange(0, per * nb + 1, per, dtype=torch.int32, device=cuda_device)
    bcols = torch.randint(0, nb, (per * nb,), device=cuda_device, generator=g, dtype=torch.int32)
    blocks = [(torch.rand(per * nb * blk * blk, device=cuda_device, generator=g) / blk).half() for _ in range(2)]
    b = torch.rand(n * feat, device=cuda_device, generator=g).half()
    ptr, cols, vals = _graph(n, 8, cuda_device, 2)

    def run(stop):
        c = torch.zeros(n * feat, device=cuda_device)
        out = [torch.zeros(n * feat, device=cuda_device) for _ in range(6)]
        torch.cuda.synchronize()
        for i, y in enumerate(out):
            ops.bsrmm(blocks[i % 2], b, c, bptr, bcols, nb, nb, per * nb, blk, feat); stop()
            ops.csrmm(vals, c, y, ptr, cols); stop()
        torch.cuda.synchronize()
        return out

    _same_without_waiting(run)


@pytest.mark.parametrize("n,feat,parts", [(3000, 32, 1), (20_000, 128, 1), (5000, 300, 1), (5000, 41, 1)])
def test_hyb_products_feed_one_another(cuda_device, n, feat, parts):
    ptr, cols, vals = _graph(n, 6, cuda_device, n + feat)
    order = torch.sort(cols.long() + torch.repeat_interleave(torch.arange(n, device=cuda_device), ptr.diff().long()) * n)[0]
    r, c, _, v, _ = fmt.column_part_hyb(n, n, ptr.cpu().numpy(), (order % n).int().cpu().numpy(), parts, (1, 2, 4, 8, 16),
                                        data=vals.cpu().numpy())
    up = lambda a: torch.from_numpy(a.reshape(-1)).to(cuda_device)  # noqa: E731
    buckets = [(up(v[0][k]), up(r[0][k]), up(c[0][k])) for k in range(5) if len(r[0][k])]
    x0 = torch.rand(n, feat, device=cuda_device)

    def run(stop):
        x, y = x0.clone(), torch.zeros_like(x0)
        there, back = ops.hyb_spmm.prepare(*ops.hyb_args(x, y, buckets, feat)), ops.hyb_spmm.prepare(*ops.hyb_args(y, x, buckets, feat))
        torch.cuda.synchronize()
        for _ in range(6):
            there(); stop()
            back(); stop()
        torch.cuda.synchronize()
        return x, y

    _same_without_waiting(run)


@pytest.mark.parametrize("n,feat", [(800, 64), (16_000, 128), (16_000, 96), (800, 512)])
def test_condensed_products_feed_one_another(cuda_device, n, feat):
    ptr, cols, _ = _graph(n, 6, cuda_device, n)
    gp, tiles, mask = fmt.condense(ptr.cpu().numpy(), cols.cpu().numpy(), 16, 16)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).to(cuda_device)  # noqa: E731
    a, gp_d, ids = up(mask).half() / 8, up(gp), up(tiles)
    x0 = torch.rand(n * feat, device=cuda_device).half()

    def run(stop):
        x, y = x0.clone(), torch.zeros_like(x0)
        torch.cuda.synchronize()
        for _ in range(5):
            ops.tcspmm(a, x, y, gp_d, ids, n // 16, n // 16, len(tiles), feat, 16, 16); stop()
            ops.tcspmm(a, y, x, gp_d, ids, n // 16, n // 16, len(tiles), feat, 16, 16); stop()
        torch.cuda.synchronize()
        return x, y

    _same_without_waiting(run)


@pytest.mark.parametrize("n,offsets,feat", [(500, 3, 64), (20_000, 8, 64), (45_000, 3, 128), (6000, 27, 256)])
def test_convolutions_feed_one_another(cuda_device, n, offsets, feat):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n)
    table = torch.randint(-n // 2, n, (-(-n // 128) * offsets * 128,), device=cuda_device, generator=g).clamp(min=-1).int()
    w = (torch.randn(offsets * feat * feat, device=cuda_device, generator=g) / (offsets * feat) ** 0.5).half()
    x0 = torch.rand(n * feat, device=cuda_device, generator=g).half() - 0.5

    def run(stop):
        x, y = x0.clone(), torch.zeros_like(x0)
        torch.cuda.synchronize()
        for add in (0, 0, 1, 0):
            ops.sparse_conv_f16(w, x, y, table, n, offsets, feat, feat, 0); stop()
            ops.sparse_conv_f16(w, y, x, table, n, offsets, feat, feat, add); stop()
        torch.cuda.synchronize()
        return x, y

    _same_without_waiting(run)


def _permutations(g, rels, feat, device, dtype):
    """A permutation matrix with signs per relation: sums of whole numbers stay whole numbers of about the same size."""
    w = torch.zeros(rels, feat, feat, device=device, dtype=dtype)
    for r in range(rels):
        sign = 2 * torch.randint(0, 2, (feat,), device=device, generator=g) - 1
        w[r, torch.arange(feat, device=device), torch.randperm(feat, device=device, generator=g)] = sign.to(dtype)
    return w.view(-1)


@pytest.mark.parametrize("n,rels,feat", [(2000, 5, 64), (30_000, 3, 64), (2000, 5, 128), (3000, 3, 256), (3000, 4, 32)])
def test_relational_layers_feed_one_another(cuda_device, n, rels, feat):
    """Layers in fp32, each adding to an output of its own.  Whole numbers: exact in any order of addition."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n + feat)
    pairs = torch.stack([torch.sort(torch.randperm(n, device=cuda_device, generator=g)[:n // 2])[0] for _ in range(rels)])
    deg = torch.randint(1, 3, (rels * (n // 2),), device=cuda_device, generator=g)
    ptr_j = torch.zeros(len(deg) + 1, dtype=torch.int32, device=cuda_device)
    ptr_j[1:] = torch.cumsum(deg, 0)
    cols = torch.randint(0, n, (int(deg.sum()),), device=cuda_device, generator=g, dtype=torch.int32)
    ptr_i = torch.arange(0, rels + 1, dtype=torch.int32, device=cuda_device) * (n // 2)
    a, w = torch.ones(len(cols), device=cuda_device), _permutations(g, rels, feat, cuda_device, torch.float32)
    x0 = torch.randint(-2, 3, (n * feat,), device=cuda_device, generator=g).float()
    rows = pairs.reshape(-1).int()

    def run(stop):
        y = [x0] + [torch.zeros_like(x0) for _ in range(5)]
        torch.cuda.synchronize()
        for x, out in zip(y, y[1:]):  # a row has at most 2 * rels terms: below 2 * 10^5 * 2 after five layers
            ops.rgms(a, w, x, out, ptr_i, rows, ptr_j, cols); stop()
        torch.cuda.synchronize()
        return y[1:]

    _same_without_waiting(run)


@pytest.mark.parametrize("widths,rows", [((1, 2), (96 << 10, 3000)), ((1,), (5000,)), ((1, 4, 2), (2000, 700, 900)), ((2,), (40_000,))])
@pytest.mark.parametrize("feat", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_half_precision_layers_feed_one_another(cuda_device, widths, rows, feat, dtype):
    """The same in fp16, whose layers take several launches that overlap; a float32 result is read by a CSR product."""
    n, rels = 2 * max(rows), 7
    g = torch.Generator(device=cuda_device)
    g.manual_seed(len(widths) + feat)
    buckets = []
    for width, count in zip(widths, rows):
        to = torch.randperm(n, device=cuda_device, generator=g)[:count].int()  # one row of a bucket per destination
        cols = torch.randint(0, n, (count * width,), device=cuda_device, generator=g, dtype=torch.int32)
        mid = torch.sort(torch.randint(0, rels, (count,), device=cuda_device, generator=g))[0].int()
        buckets.append((torch.ones(count * width, device=cuda_device, dtype=torch.float16), to, cols, mid))
    w = _permutations(g, rels, feat, cuda_device, torch.float16)
    x0 = torch.randint(-2, 3, (n * feat,), device=cuda_device, generator=g).half()
    ptr, cols, vals = _graph(n, 3, cuda_device, n)

    def run(stop):
        torch.cuda.synchronize()
        if dtype == torch.float16:  # at most 2 * 7^3 in three layers: exact
            y = [x0] + [torch.zeros_like(x0) for _ in range(3)]
            torch.cuda.synchronize()
            for x, out in zip(y, y[1:]):
                ops.rgms_ell3d_f16(*ops.rgms_ell3d_f16_args(w, x, out, buckets, feat, feat)); stop()
            torch.cuda.synchronize()
            return y[1:]
        y, z = torch.zeros(n * feat, device=cuda_device), [torch.zeros(n * feat, device=cuda_device) for _ in range(4)]
        torch.cuda.synchronize()
        for out in z:  # the next layer adds to what the CSR product reads
            ops.rgms_ell3d_f16(*ops.rgms_ell3d_f16_args(w, x0, y, buckets, feat, feat)); stop()
            ops.csrmm(vals, y, out, ptr, cols); stop()
        torch.cuda.synchronize()
        return [y] + z

    _same_without_waiting(run)
