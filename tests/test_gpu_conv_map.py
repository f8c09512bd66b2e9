"""The sparse convolution with its neighbour map laid out in advance: channel counts around the
slices and boxes of the kernel, ragged tiles, offsets without pairs, and addition into an output."""
import numpy as np
import pytest
import torch

from sparsetir_b200 import _lib as L
from sparsetir_b200 import ops
from sparsetir_b200.sparse_conv import SparseConvPlan, neighbour_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("feat_in", [16, 32, 48, 64, 96, 128, 256])
@pytest.mark.parametrize("feat_out", [32, 64, 96, 160, 256])
@pytest.mark.parametrize("n_out,offsets,fill", [(1, 1, 1.0), (127, 3, 0.5), (129, 27, 0.3), (20_001, 8, 0.6)])
def test_matches_a_float64_product(cuda_device, feat_in, feat_out, n_out, offsets, fill):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(feat_in + feat_out + n_out)
    n_in = max(2, n_out // 2)
    maps, sizes = [], []
    for k in range(offsets):
        outs = torch.nonzero(torch.rand(n_out, device=cuda_device, generator=g) < (0.0 if k == 1 else fill))[:, 0]
        ins = torch.randint(0, n_in, (len(outs),), device=cuda_device, generator=g)
        maps.append(torch.stack([ins, outs], 1))
        sizes.append(len(outs))
    pairs = torch.cat(maps)
    x = torch.rand(n_in, feat_in, device=cuda_device, generator=g).half() - 0.5
    w = (torch.randn(offsets, feat_in, feat_out, device=cuda_device, generator=g) / np.sqrt(feat_in)).half()
    table = neighbour_map(pairs, np.asarray(sizes), False, n_out, cuda_device)
    want = torch.zeros(n_out, feat_out, dtype=torch.float64, device=cuda_device)
    mag = torch.zeros_like(want)
    for k, mp in enumerate(maps):
        want[mp[:, 1]] += x[mp[:, 0]].double() @ w[k].double()
        mag[mp[:, 1]] += x[mp[:, 0]].double().abs() @ w[k].double().abs()
    # fp32 sums of exact fp16 products (the tensor core may cut below the last bit of the largest
    # term of every 16-term step: one ulp a step); the start value and a float16 result round once more
    bound = mag * (offsets * feat_in / 16 + 2) * 2.0 ** -22
    for dtype, add in ((torch.float32, 0), (torch.float32, 1), (torch.float16, 0), (torch.float16, 1)):
        y = torch.full((n_out * feat_out,), 3.0, dtype=dtype, device=cuda_device)
        ops.sparse_conv_f16(w.view(-1), x.view(-1), y, table, n_out, offsets, feat_in, feat_out, add)
        ref = want + 3.0 * add
        extra = ref.abs() * 2.0 ** -22 if dtype == torch.float32 else (ref.abs() + want.abs()) * 2.0 ** -10 + 2.0 ** -20
        assert bool(((y.view(n_out, feat_out).double() - ref).abs() <= bound + extra).all()), (dtype, add)
    count = L.ctypes.c_uint(0)
    assert L.load().sparsetir_tc_timeouts(cuda_device.index or 0, L.ctypes.byref(count)) == 0 and count.value == 0


@pytest.mark.parametrize("feat_in,feat_out", [(64, 128), (48, 96), (16, 32), (64, 160)])
@pytest.mark.parametrize("n_out", [7, 8, 9, 1185, 18_943, 18_945, 37_889, 60_007])
@pytest.mark.parametrize("shift", [0, 1])
def test_shares_of_blocks_and_maps_that_are_not_aligned(cuda_device, feat_in, feat_out, n_out, shift):
    """Tiles of a few rows, blocks with one tile and with two side by side, an odd one left over; a map whose entries are not
    16-byte aligned."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n_out + feat_in)
    offsets = 3
    table = torch.full((-(-n_out // 128) * offsets * 128 + shift,), -1, dtype=torch.int32, device=cuda_device)[shift:]
    x = torch.rand(500, feat_in, device=cuda_device, generator=g).half() - 0.5
    w = torch.randn(offsets, feat_in, feat_out, device=cuda_device, generator=g).half() / 8
    want = torch.zeros(n_out, feat_out, dtype=torch.float64, device=cuda_device)
    mag = torch.zeros_like(want)
    for k in range(offsets):
        src = torch.randint(-300, 500, (n_out,), device=cuda_device, generator=g).clamp(min=-1)
        at = torch.arange(n_out, device=cuda_device)
        table[(at // 128 * offsets + k) * 128 + at % 128] = src.int()
        rows = x.double()[src.clamp(min=0)] * (src >= 0)[:, None]
        want += rows @ w[k].double()
        mag += rows.abs() @ w[k].double().abs()
    y = torch.full((n_out * feat_out + 32,), 3.0, device=cuda_device)
    ops.sparse_conv_f16(w.view(-1), x.view(-1), y[:n_out * feat_out], table, n_out, offsets, feat_in, feat_out, 0)
    bound = mag * (offsets * feat_in / 16 + 2) * 2.0 ** -22  # as above
    assert bool(((y[:-32].view(n_out, feat_out).double() - want).abs() <= bound).all())
    assert bool((y[-32:] == 3.0).all())


@pytest.mark.parametrize("feat_in,feat_out", [(64, 128), (32, 64), (128, 256)])
def test_the_same_bits_on_every_call(cuda_device, feat_in, feat_out):
    """Copies of a stage arrive at its barrier by themselves: nothing of a stage may be read before it has landed."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(feat_in)
    n, offsets = 50_000, 27
    src = torch.randint(-n // 2, n, (-(-n // 128) * offsets * 128,), device=cuda_device, generator=g).clamp(min=-1).int()
    x = (torch.randint(-2, 3, (n, feat_in), device=cuda_device, generator=g)).half()
    w = (torch.randint(-2, 3, (offsets, feat_in, feat_out), device=cuda_device, generator=g)).half()
    want = torch.zeros(n, feat_out, device=cuda_device)
    table = src.view(-1, offsets, 128)
    for k in range(offsets):  # whole numbers below 2^24: exact in any order
        s = table[:, k].reshape(-1)[:n].long()
        want += torch.where((s >= 0)[:, None], x[s.clamp(min=0)].float(), 0.0) @ w[k].float()
    y = torch.empty(n * feat_out, device=cuda_device)
    for _ in range(30):
        y.fill_(7.0)
        ops.sparse_conv_f16(w.view(-1), x.view(-1), y, src, n, offsets, feat_in, feat_out, 0)
        assert torch.equal(y.view(n, feat_out), want)


@pytest.mark.parametrize("feat_in,feat_out", [(64, 128), (48, 96), (16, 32), (64, 160)])
@pytest.mark.parametrize("n_out", [5, 18_943, 18_945, 37_889, 60_007])
@pytest.mark.parametrize("dtype,add", [(torch.float16, 0), (torch.float16, 1), (torch.float32, 1)])
def test_two_tiles_a_stage_in_both_types_and_added(cuda_device, feat_in, feat_out, n_out, dtype, add):
    """The forms of the test above with a float16 result and with addition into the output: whole numbers, exact in both."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n_out + feat_in)
    offsets = 3
    table = torch.full((-(-n_out // 128) * offsets * 128,), -1, dtype=torch.int32, device=cuda_device)
    x = torch.randint(-1, 2, (500, feat_in), device=cuda_device, generator=g).half()
    w = torch.randint(-1, 2, (offsets, feat_in, feat_out), device=cuda_device, generator=g).half()
    y = torch.randint(-5, 6, (n_out * feat_out + 32,), device=cuda_device, generator=g).to(dtype)
    want = y[:-32].view(n_out, feat_out).double() * add
    for k in range(offsets):
        src = torch.randint(-300, 500, (n_out,), device=cuda_device, generator=g).clamp(min=-1)
        at = torch.arange(n_out, device=cuda_device)
        table[(at // 128 * offsets + k) * 128 + at % 128] = src.int()
        want += (x.double()[src.clamp(min=0)] * (src >= 0)[:, None]) @ w[k].double()
    behind = y[-32:].clone()
    ops.sparse_conv_f16(w.view(-1), x.view(-1), y[:n_out * feat_out], table, n_out, offsets, feat_in, feat_out, add)
    assert torch.equal(y[:-32].view(n_out, feat_out).double(), want) and torch.equal(y[-32:], behind)


def test_weights_that_are_not_finite_reach_their_own_pairs_only(cuda_device):
    n, pairs = 300, torch.tensor([[5, 7], [9, 7], [2, 299]])
    x = torch.full((n, 32), 0.5, device=cuda_device).half()
    w = torch.full((2, 32, 64), 0.25, device=cuda_device).half()
    w[1, 3, 40] = float("inf")
    want = torch.zeros(n, 64, device=cuda_device)
    want[7], want[299] = 8.0, 4.0
    want[7, 40] = want[299, 40] = float("inf")
    table = neighbour_map(pairs, [1, 2], False, n, cuda_device)
    y = torch.empty(n * 64, device=cuda_device)
    ops.sparse_conv_f16(w.view(-1), x.view(-1), y, table, n, 2, 32, 64, 0)
    assert torch.equal(y.view(n, 64), want)


def test_repeated_pairs_keep_the_buckets(cuda_device):
    pairs = torch.tensor([[0, 1], [2, 1], [1, 0]])
    assert neighbour_map(pairs, [2, 1], False, 3, cuda_device) is None
    x, w = torch.rand(3, 64, device=cuda_device).half(), torch.rand(2, 64, 64, device=cuda_device).half()
    y = SparseConvPlan(pairs, [2, 1], False, 3, 3, device=cuda_device)(x, w, out_dtype=torch.float32)
    want = torch.zeros(3, 64, device=cuda_device)
    want[1] = (x[0].float() + x[2].float()) @ w[0].float()
    want[0] = x[1].float() @ w[1].float()
    torch.testing.assert_close(y, want, rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("nbmaps,sizes", [(np.zeros((0, 2), np.int64), []), (np.zeros((0, 2), np.int64), [0, 0]),
                                          (np.array([[0, 1], [2, 1], [1, 0]])[:, ::-1], [2, 1])])
@pytest.mark.parametrize("feat_in,feat_out", [(64, 128), (256, 64), (32, 48)])
def test_plans_of_few_pairs(cuda_device, nbmaps, sizes, feat_in, feat_out):
    x = torch.rand(3, feat_in, device=cuda_device).half()
    w = torch.rand(len(sizes), feat_in, feat_out, device=cuda_device).half() / 16
    y = SparseConvPlan(nbmaps, sizes, True, 3, 3, device=cuda_device)(x, w, out_dtype=torch.float32)
    want, at = torch.zeros(3, feat_out, dtype=torch.float64, device=cuda_device), 0
    for k, size in enumerate(sizes):
        for o, i in nbmaps[at:at + size].tolist():
            want[o] += x[i].double() @ w[k].double()
        at += size
    torch.testing.assert_close(y.double(), want, rtol=1e-5, atol=1e-5)


def test_shapes_it_does_not_take_are_refused(cuda_device):
    h = lambda n: torch.zeros(n, dtype=torch.float16, device=cuda_device)  # noqa: E731
    table = torch.full((128,), -1, dtype=torch.int32, device=cuda_device)
    for fi, fo in ((8, 32), (16, 16), (16, 288)):
        with pytest.raises(ops.SparseTIRError, match="multiple of 16"):
            ops.sparse_conv_f16(h(fi * fo), h(fi), h(fo), table, 1, 1, fi, fo, 0)
    with pytest.raises(ops.SparseTIRError, match="map"):
        ops.sparse_conv_f16(h(32 * 32), h(32), h(32), table[:64], 1, 1, 32, 32, 0)
