"""Calls whose time must follow the work in them: rows of very different lengths beside rows of one length, fewer features beside
more.  A ratio of two times, taken in turn on the same GPU; every limit lies well above what is measured."""
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


def csr_call(f, device, deg, feat):
    """A kept call of sddmm or csrmm on a matrix of uniformly drawn columns."""
    n, nnz = len(deg), int(deg.sum())
    g = torch.Generator(device=device).manual_seed(feat)
    ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).to(device)
    cols = torch.randint(0, n, (nnz,), generator=g, device=device, dtype=torch.int32)
    a, b, e = (torch.rand(k, generator=g, device=device) for k in (n * feat, n * feat, nnz))
    return f.prepare(a, b, e, ptr, cols) if f is ops.sddmm else f.prepare(e, a, b, ptr, cols)


@pytest.mark.parametrize("n,mean,feat,limit", [(100_000, 30, 256, 1.2), (20_000, 30, 24, 1.18)])
def test_sddmm_on_uneven_rows(cuda_device, n, mean, feat, limit):
    uneven = lengths("uneven", n, mean)
    even = lengths("equal", n, int(round(uneven.sum() / n)))
    check_ratio(csr_call(ops.sddmm, cuda_device, uneven, feat), csr_call(ops.sddmm, cuda_device, even, feat), limit)


@pytest.mark.parametrize("op,n,mean,feat,other,limit", [
    ("sddmm", 20_000, 10, 512, 128, 3.85), ("sddmm", 20_000, 100, 224, 256, 1.08), ("sddmm", 10_000, 11, 40, 64, 1.3), ("sddmm", 80_000, 5, 298, 300, 1.4),
    ("csrmm", 10_000, 4, 512, 256, 1.62), ("csrmm", 20_000, 3, 384, 256, 1.4)])
def test_more_and_fewer_features(cuda_device, op, n, mean, feat, other, limit):
    """Beside a neighbour that is known to be served well: what is fixed in a call weighs less where there are more features."""
    deg, f = lengths("equal", n, mean), getattr(ops, op)
    check_ratio(csr_call(f, cuda_device, deg, feat), csr_call(f, cuda_device, deg, other), limit)


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
    check_ratio(layer(hubs), layer(np.full(10_000, 8, np.int64)), 2.0)


@pytest.mark.parametrize("n,width,feat,other,limit", [(20_000, 4, 299, 300, 1.13), (20_000, 8, 512, 256, 2.2)])
def test_hyb_of_more_and_fewer_features(cuda_device, n, width, feat, other, limit):
    """ELL rows of one width."""
    def call(f):
        g = torch.Generator(device=cuda_device).manual_seed(f)
        x = torch.rand(n, f, generator=g, device=cuda_device)
        bucket = (torch.rand(n * width, generator=g, device=cuda_device), torch.arange(n, device=cuda_device, dtype=torch.int32),
                  torch.randint(0, n, (n * width,), generator=g, device=cuda_device, dtype=torch.int32))
        return ops.hyb_spmm.prepare(*ops.hyb_args(x, torch.zeros(n, f, device=cuda_device), [bucket], f, 0))
    check_ratio(call(feat), call(other), limit)


def test_rgms_f16_with_more_ranges_than_a_block_keeps(cuda_device):
    """1,800 (bucket, relation) ranges, most of them empty, beside 900."""
    def layer(rels, n=2000, feat=32):
        g = torch.Generator(device=cuda_device).manual_seed(rels)
        buckets = []
        for width in (1, 2, 4, 8, 16, 32):
            k = rels if width == 1 else 2
            shape = (k, 32 // width, width)
            buckets.append((torch.rand(shape, generator=g, device=cuda_device).half(),
                            torch.randint(0, n, shape[:2], generator=g, device=cuda_device).int(),
                            torch.randint(0, n, shape, generator=g, device=cuda_device).int(), torch.arange(k, device=cuda_device).int()))
        x, w = (torch.rand(k, generator=g, device=cuda_device).half() for k in (n * feat, rels * feat * feat))
        return ops.rgms_ell3d_f16.prepare(*ops.rgms_ell3d_f16_args(w, x, torch.zeros(n * feat, device=cuda_device), buckets, feat, feat))
    check_ratio(layer(300), layer(150), 3.45)
