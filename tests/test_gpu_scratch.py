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


CALLS = {"csrmm": csrmm_call, "tcspmm": tcspmm_call}


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
