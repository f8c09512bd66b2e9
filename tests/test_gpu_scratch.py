"""Operator calls and the library's scratch memory: calls that are captured into a graph, and calls whose
stages hold scratch at the same time."""
import ctypes

import numpy as np
import pytest
import torch

from sparsetir_b200 import _lib as L
from sparsetir_b200 import format as fmt
from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


def csr(device, m, n, mean, seed=0):
    """Row lengths around `mean`, one hub row, rows without entries: row ends anywhere in a block."""
    rng = np.random.default_rng(seed)
    deg = rng.poisson(mean, m)
    deg[:3] = [min(n, 5000), 0, min(n, 700)]
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    cols = rng.integers(0, n, int(ptr[-1])).astype(np.int32)
    return torch.from_numpy(ptr).to(device), torch.from_numpy(cols).to(device)


def csrmm_call(device, feat):
    ptr, cols = csr(device, 9000, 4000, 9)
    vals, x = torch.rand(len(cols), device=device), torch.rand(4000 * feat, device=device)
    y = torch.empty(9000 * feat, device=device)
    return y, lambda: ops.csrmm(vals, x, y, ptr, cols)


def tcspmm_call(device, feat):
    rng = np.random.default_rng(1)
    deg = np.zeros(6000, np.int64)
    deg[[8, 40, 4000]] = [5900, 3000, 300]  # tiles over several windows
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(6000, d, replace=False)) for d in deg]).astype(np.int32)
    gp, tiles, mask = fmt.condense(ptr, cols, 16, 16)
    up = lambda t: torch.from_numpy(np.ascontiguousarray(t).reshape(-1)).to(device)  # noqa: E731
    a, gp, ids, x = up(mask).half(), up(gp), up(tiles), torch.rand(6000 * feat, device=device).half()
    y = torch.empty(6000 * feat, device=device)
    return y, lambda: ops.tcspmm(a, x, y, gp, ids, 375, 375, len(tiles), feat, 16, 16)


def hyb_call(device, feat):
    ptr, cols = (t.cpu().numpy() for t in csr(device, 3000, 4000, 5))
    r, c, _, v, _ = fmt.column_part_hyb(3000, 4000, ptr, cols, 1, [1, 2, 4, 8, 16, 32],
                                        data=np.random.default_rng(0).random(len(cols), np.float32))
    up = lambda t: torch.from_numpy(np.ascontiguousarray(t).reshape(-1)).to(device)  # noqa: E731
    buckets = [(up(v[0][b]), up(r[0][b]), up(c[0][b])) for b in range(6) if len(r[0][b])]
    x, y = torch.rand(4000 * feat, device=device), torch.zeros(3000 * feat, device=device)
    return y, lambda: ops.hyb_spmm(*ops.hyb_args(x, y, buckets, feat))


CALLS = {"csrmm": csrmm_call, "tcspmm": tcspmm_call}


def fresh_stream():
    """A stream without buffers: of the high-priority pool, which hands out 32 before it repeats."""
    return torch.cuda.Stream(priority=-1)


def grow_buffers(stream):
    """Makes the library give up the buffers that the stream has for larger ones."""
    assert L.load().sparsetir_reserve_workspace(0, ctypes.c_void_p(stream.cuda_stream), 48 << 20, 4 << 20) == 0


@pytest.mark.parametrize("op", sorted(CALLS))
@pytest.mark.parametrize("feat", [64, 136])
def test_a_graph_outlives_the_buffers_of_its_stream(cuda_device, op, feat):
    y, call = CALLS[op](cuda_device, feat)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):  # the stream has buffers that fit the call
        call()
    stream.synchronize()
    want = y.clone()
    with torch.cuda.graph(graph, stream=stream):
        call()
    grow_buffers(stream)
    for _ in range(2):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)


@pytest.mark.parametrize("op", sorted(CALLS))
@pytest.mark.parametrize("captured", [False, True])
def test_calls_on_two_streams_at_once(cuda_device, op, captured):
    # eager calls use the buffers of their own stream; replays, also of two graphs that were captured
    # on one stream, use memory of their own
    pairs = [CALLS[op](cuda_device, 64) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    want, graphs = [], []
    for y, call in pairs:
        with torch.cuda.stream(streams[0]):
            call()
        streams[0].synchronize()
        want.append(y.clone())
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=streams[0]):
            call()
        y.zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for stream, graph, (y, call) in zip(streams, graphs, pairs):
            with torch.cuda.stream(stream):
                graph.replay() if captured else call()
    torch.cuda.synchronize()
    for (y, _), w in zip(pairs, want):
        assert torch.equal(y, w)


@pytest.mark.parametrize("feat", [41, 100, 130])
def test_the_first_hyb_call_on_a_stream_can_be_captured(cuda_device, feat):
    y, call = hyb_call(cuda_device, feat)
    call()
    want, graph, stream = y.clone(), torch.cuda.CUDAGraph(), fresh_stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        call()
    grow_buffers(stream)
    for _ in range(2):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)


def test_captured_rgms_outlives_the_buffers_of_its_stream(cuda_device):
    n, rels, per, feat = 600, 4, 900, 128
    g = torch.Generator(device=cuda_device)
    g.manual_seed(0)
    pair = torch.sort(torch.stack([torch.randperm(n, device=cuda_device, generator=g)[:300] for _ in range(rels)]), 1)[0]
    ptr_i = torch.arange(0, rels * 300 + 1, 300, dtype=torch.int32, device=cuda_device)
    ptr_j = torch.arange(0, rels * per + 1, per // 300, dtype=torch.int32, device=cuda_device)
    src = torch.randint(0, n, (rels * per,), dtype=torch.int32, device=cuda_device, generator=g)
    a, w, x = (torch.rand(k, device=cuda_device, generator=g) for k in (rels * per, rels * feat * feat, n * feat))
    y = torch.zeros(n * feat, device=cuda_device)
    rows = pair.reshape(-1).int()
    call = lambda: ops.rgms(a, w, x, y, ptr_i, rows, ptr_j, src)  # noqa: E731
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        call()
    stream.synchronize()
    want = y.clone()
    with torch.cuda.graph(graph, stream=stream):
        call()
    grow_buffers(stream)
    for _ in range(2):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        # fp32 sums of at most 4 rows of terms that are not negative, added in any order
        torch.testing.assert_close(y, want, rtol=8 * 2.0 ** -24, atol=0)


def attention_float64(q, k, v, ptr, cols):
    """(result, bound of the error of fp32 stages in any order).  The numerator is not shifted by the row maximum:
    exp(s) / sum exp(s - max), as in the reference (tests/refimpl.py)."""
    (m, feat), n = q.shape, k.shape[0]
    deg = (ptr[1:] - ptr[:-1]).long()
    rows = torch.repeat_interleave(torch.arange(m, device=q.device), deg)
    s, mag = (torch.cat([(x[rows[p:p + 50_000]] * y[cols[p:p + 50_000].long()]).sum(1) for p in range(0, len(cols), 50_000)])
              for x, y in ((q.double(), k.double()), (q.abs().double(), k.abs().double())))
    top = torch.full((m,), -float("inf"), dtype=torch.float64, device=q.device).scatter_reduce(0, rows, s, "amax")
    total = torch.zeros(m, dtype=torch.float64, device=q.device).index_add_(0, rows, torch.exp(s - top[rows]))
    prob = torch.exp(s) / total[rows]
    out, size = (torch.zeros(m, feat, dtype=torch.float64, device=q.device) for _ in range(2))
    for p in range(0, len(cols), 50_000):
        part = prob[p:p + 50_000, None] * v[cols[p:p + 50_000].long()].double()
        out.index_add_(0, rows[p:p + 50_000], part)
        size.index_add_(0, rows[p:p + 50_000], part.abs())
    # a score is off by feat half-ulps of its terms, which becomes a relative error of its exponential (two
    # scores: its own and the maximum); __expf(x) adds 2 + 1.2 |x| ulps with |x| up to twice the largest
    # score; row sum, quotient and weighted sum add (entries of the row + a few) half-ulps
    score = 2 * float(mag.max()) * (feat + 2) * 2.0 ** -24 + (6 + 2.4 * float(s.abs().max())) * 2.0 ** -23
    return out, size * (2 * score + (2 * deg[:, None].double() + 16) * 2.0 ** -24)


@pytest.mark.parametrize("feat", [128, 256, 300, 500, 512])
@pytest.mark.parametrize("m,mean", [(19_717, 4), (50_000, 6), (2_000, 50)])
def test_attention_keeps_its_probabilities_beside_the_pieces(cuda_device, feat, m, mean):
    # the SpMM stage splits rows over blocks and needs scratch while the scratch of the stage before is its operand
    ptr, cols = csr(cuda_device, m, m, mean, seed=feat)
    q, k, v = (torch.rand(m, feat, device=cuda_device) * 2 - 1 for _ in range(3))
    q *= 2.0 / feat ** 0.5
    want, bound = attention_float64(q, k, v, ptr, cols)
    o = torch.full((m * feat,), float("nan"), device=cuda_device)
    call = lambda: ops.fusedmm(q.view(-1), k.view(-1), v.view(-1), o, ptr, cols)  # noqa: E731
    stream, graph = fresh_stream(), torch.cuda.CUDAGraph()  # its buffers come out as small as asked for
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        call()
    stream.synchronize()
    assert bool(((o.view(m, feat).double() - want).abs() <= bound).all())
    first = o.clone()
    with torch.cuda.stream(stream):
        call()
    stream.synchronize()
    assert torch.equal(first, o)
    with torch.cuda.graph(graph, stream=stream):
        call()
    o.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(first, o)


@pytest.mark.parametrize("feat", [100, 256, 41])
def test_calls_on_a_reserved_stream_allocate_nothing(cuda_device, feat):
    lib, stream = L.load(), fresh_stream()
    m = n = 20_000
    ptr, cols = csr(cuda_device, m, n, 12)
    nnz = len(cols)
    vals, q, k, v, o = (torch.rand(size, device=cuda_device) for size in (nnz, m * feat, n * feat, n * feat, m * feat))
    calls = [(("sparsetir_csrmm_workspace", m, n, feat, nnz), lambda: ops.csrmm(vals, v, o, ptr, cols)),
             (("sparsetir_fusedmm_workspace", m, n, nnz, feat), lambda: ops.fusedmm(q, k, v, o, ptr, cols))]
    groups, t = 3000, 16
    a = torch.ones(groups * t * 16, device=cuda_device, dtype=torch.float16)
    gp = torch.tensor([0, 2900, 2900, groups], dtype=torch.int32, device=cuda_device)
    ids = torch.arange(groups * 16, device=cuda_device).remainder(n).int()
    b, c = torch.rand(n * 64, device=cuda_device).half(), torch.empty(3 * t * 64, device=cuda_device)
    calls.append((("sparsetir_tcspmm_workspace", groups, 64, t, 16), lambda: ops.tcspmm(a, b, c, gp, ids, 3, n // 16, groups, 64, t, 16)))
    for (query, *sizes), call in calls:
        need = [ctypes.c_size_t(0) for _ in range(2)]
        assert getattr(lib, query)(*sizes, *(ctypes.byref(x) for x in need)) == 0
        assert lib.sparsetir_reserve_workspace(0, ctypes.c_void_p(stream.cuda_stream), *need) == 0
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        with torch.cuda.stream(stream):
            call()
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
