"""Calls whose time must follow the work in them: rows of very different lengths beside rows of one length, fewer features beside
more.  A ratio of two times, taken in turn on the same GPU.  The same ratio differs by up to 7 % from one GPU to another, so only
faults that are a factor have a test: a limit lies about midway, in factors, between what the call takes and what it took with the fault."""
import numpy as np
import pytest
import torch

from sparsetir_b200 import ops

pytestmark = pytest.mark.gpu


def times(calls, rounds=7):
    """us of each call among others like it: the median of rounds that take the calls in turn."""
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    reps = []
    for call in calls:
        for _ in range(3):
            call()
        begin.record()
        call()
        end.record()
        end.synchronize()
        reps.append(int(min(200, max(5, 2.0 / max(begin.elapsed_time(end), 1e-3)))))
    out = [[] for _ in calls]
    for _ in range(rounds):
        for i, call in enumerate(calls):
            call()
            begin.record()
            for _ in range(reps[i]):
                call()
            end.record()
            end.synchronize()
            out[i].append(begin.elapsed_time(end) / reps[i] * 1e3)
    return [sorted(t)[rounds // 2] for t in out]


def check_ratio(call, other, limit):
    """call takes at most `limit` times as long as other; a GPU that was busy gets two more chances."""
    seen = []
    for _ in range(3):
        t, u = times([call, other])
        seen.append(t / u)
        if seen[-1] <= limit:
            return
    pytest.fail(f"{seen} against {limit}")


def lengths(kind, n, mean):
    if kind == "equal":
        return np.full(n, mean, np.int64)
    rng = np.random.default_rng(n)  # log-normal of sigma 2: half of the rows have less than a seventh of the mean
    return np.clip(np.rint(rng.lognormal(np.log(mean) - 2.0, 2.0, n)), 1, n // 4).astype(np.int64)


def sddmm_call(device, deg, feat):
    """A kept call on a matrix of uniformly drawn columns."""
    n, nnz = len(deg), int(deg.sum())
    g = torch.Generator(device=device).manual_seed(feat)
    ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).to(device)
    cols = torch.randint(0, n, (nnz,), generator=g, device=device, dtype=torch.int32)
    a, b, e = (torch.rand(k, generator=g, device=device) for k in (n * feat, n * feat, nnz))
    return ops.sddmm.prepare(a, b, e, ptr, cols)


@pytest.mark.parametrize("n,mean,feat,limit", [(100_000, 30, 256, 1.2), (20_000, 30, 24, 1.22)])
def test_sddmm_on_uneven_rows(cuda_device, n, mean, feat, limit):
    uneven = lengths("uneven", n, mean)
    even = lengths("equal", n, int(round(uneven.sum() / n)))
    check_ratio(sddmm_call(cuda_device, uneven, feat), sddmm_call(cuda_device, even, feat), limit)


@pytest.mark.parametrize("feat", [64, 128])
def test_rgms_with_hub_destinations(cuda_device, feat):
    """20 of 10,000 destinations with 2,000 edges each, beside as many edges evenly."""
    def layer(deg):
        n, nnz = len(deg), int(deg.sum())
        g = torch.Generator(device=cuda_device).manual_seed(feat)
        ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).to(cuda_device)
        cols = torch.randint(0, n, (nnz,), generator=g, device=cuda_device, dtype=torch.int32)
        a, w, x = (torch.rand(k, generator=g, device=cuda_device) for k in (nnz, feat * feat, n * feat))
        rows = torch.arange(n, device=cuda_device, dtype=torch.int32)
        return ops.rgms.prepare(a, w, x, torch.zeros(n * feat, device=cuda_device), torch.tensor([0, n], device=cuda_device, dtype=torch.int32), rows,
                                ptr, cols)
    hubs = np.full(10_000, 4, np.int64)
    hubs[250::500] = 2_000
    check_ratio(layer(hubs), layer(np.full(10_000, 8, np.int64)), 4.4)


def test_hyb_of_more_features(cuda_device, n=20_000, width=8, feat=512, other=256, limit=2.0):
    """ELL rows of one width."""
    def call(f):
        g = torch.Generator(device=cuda_device).manual_seed(f)
        x = torch.rand(n, f, generator=g, device=cuda_device)
        bucket = (torch.rand(n * width, generator=g, device=cuda_device), torch.arange(n, device=cuda_device, dtype=torch.int32),
                  torch.randint(0, n, (n * width,), generator=g, device=cuda_device, dtype=torch.int32))
        return ops.hyb_spmm.prepare(*ops.hyb_args(x, torch.zeros(n, f, device=cuda_device), [bucket], f, 0))
    check_ratio(call(feat), call(other), limit)
