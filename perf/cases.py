"""The sparse operators as programs use them: one case is one call of a public operator of
``sparsetir_b200`` on one matrix, at sizes from a few thousand rows to the largest graph of the
benchmark configurations.

``listed()`` holds the named cases, ``draw(rng)`` gives further ones of the same ranges.  A case is
a flat dict: ``op`` names the operator, the rest are its sizes and options.

``call`` says how the program calls: ``"each"`` passes the tensors on every call (a layer of a
network, whose activations are other tensors each time), ``"kept"`` keeps the packed call of fixed
buffers (``PackedFunc.prepare``: an iterative method, a serving loop with static buffers).

The number of stored entries of a case is fixed (its degree sequence comes from the sizes alone);
which row has which degree, the columns, the values and the dense operands come from the seed.
"""
import math

import numpy as np
import torch

from sparsetir_b200 import format as fmt
from sparsetir_b200 import ops
from sparsetir_b200.sparse_conv import SparseConvPlan

HYB_WIDTHS = (1, 2, 4, 8, 16, 32, 64, 128, 256, 512)


def listed():
    return [
        # the smallest call: a 4096-row matrix, where the launch and the host path count
        dict(name="csr_spmm_small", op="csr_spmm", degrees="poisson", n=4096, mean=10.0, feat=64, call="each"),
        # a graph with hub rows used as it comes, without a format conversion; ragged sizes
        dict(name="csr_spmm_graph", op="csr_spmm", degrees="powerlaw", n=100_003, mean=0.0, feat=100, call="each"),
        # neighbour aggregation on the power-law graph in the hyb format: the narrow output layer ...
        dict(name="hyb_spmm_narrow", op="hyb_spmm", degrees="powerlaw", n=169_343, mean=0.0, feat=32, parts=1, call="each"),
        # ... and the widest layer
        dict(name="hyb_spmm_wide", op="hyb_spmm", degrees="powerlaw", n=169_343, mean=0.0, feat=512, parts=1, call="kept"),
        # edge scores on the same graph: also what the gradient of SpMM with respect to A computes
        dict(name="sddmm_graph", op="sddmm", degrees="powerlaw", n=169_343, mean=0.0, feat=64, call="each"),
        # edge scores on the largest graph: 1.2e8 stored positions
        dict(name="sddmm_large", op="sddmm", degrees="lognormal", n=232_965, mean=0.0, feat=128, call="kept"),
        # sparse attention with a block mask: fp16 blocks, fp32 result
        dict(name="bsr_attention", op="bsrmm", n=4096, blk=32, density=0.10, feat=512, call="each"),
        # one relational layer (46 relations, 1.5 M edges), fp32
        dict(name="rgms_fp32", op="rgms", n=100_000, rels=46, edges=1_500_000, feat=64, call="each"),
        # the same layer in fp16 on ELL3D buckets (the tensor-core RGCN operator)
        dict(name="rgcn_fp16", op="rgcn_f16", n=100_000, rels=46, edges=1_500_000, feat_in=64, feat_out=64, call="each"),
        # a 3x3x3 sparse convolution layer on 100,000 points, through its plan
        dict(name="sparse_conv", op="sparse_conv", n=100_000, offsets=27, fill=0.5926, feat_in=64, feat_out=128),
        # attention restricted to the edges of a graph: scores, softmax and weighted sum
        dict(name="graph_attention", op="fusedmm", degrees="lognormal", n=40_000, mean=0.0, feat=64, call="each"),
        # fp16 SpMM on the condensed format
        dict(name="tc_spmm", op="tcspmm", degrees="powerlaw", n=169_343, mean=0.0, feat=128, call="kept"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["csr_spmm", "hyb_spmm", "hyb_spmm", "sddmm", "bsrmm", "rgms", "rgcn_f16", "sparse_conv",
                     "fusedmm", "tcspmm"])
    call = rng.choice(["each", "each", "kept"])
    if op in ("csr_spmm", "hyb_spmm", "sddmm"):
        degrees = rng.choice(["poisson", "powerlaw"])
        c = dict(op=op, degrees=degrees, n=_log_int(rng, 3_000, 200_000),
                 mean=round(rng.uniform(4.0, 40.0), 1) if degrees == "poisson" else 0.0,
                 feat=rng.choice([32, 64, 128, 256, 512, 4 * rng.randint(4, 75), rng.randint(17, 300)]), call=call)
        if op == "hyb_spmm":
            c["parts"] = rng.choice([1, 1, 1, 2])
        return c
    if op == "bsrmm":
        blk = rng.choice([16, 32, 32, 64])
        return dict(op=op, n=blk * (_log_int(rng, 1024, 8192) // blk), blk=blk, density=round(rng.uniform(0.02, 0.2), 3),
                    feat=rng.choice([64, 128, 256, 512, 16 * rng.randint(2, 32)]), call=call)
    if op in ("rgms", "rgcn_f16"):
        n = _log_int(rng, 3_000, 100_000)
        c = dict(op=op, n=n, rels=rng.randint(4, 90), edges=int(n * rng.uniform(4.0, 15.0)), call=call)
        if op == "rgms":
            return dict(c, feat=rng.choice([32, 64, 64, 64, 128]))
        return dict(c, feat_in=rng.choice([32, 64, 64, 128]), feat_out=rng.choice([32, 64, 64, 128]))
    if op == "sparse_conv":
        fi, fo = rng.choice([32, 64, 96, 128]), rng.choice([32, 64, 96, 128, 256])
        # the layers with more channels are those with fewer points
        return dict(op=op, n=_log_int(rng, 4_000, min(100_000, 100_000 * 64 * 128 // (fi * fo))), offsets=rng.choice([8, 27, 27]),
                    fill=round(rng.uniform(0.2, 0.6), 2), feat_in=fi, feat_out=fo)
    if op == "fusedmm":
        return dict(op=op, degrees="lognormal", n=_log_int(rng, 2_000, 40_000), mean=0.0,
                    feat=rng.choice([32, 64, 64, 128, 8 * rng.randint(3, 16)]), call=call)
    return dict(op=op, degrees="powerlaw", n=_log_int(rng, 3_000, 169_343), mean=0.0,
                feat=rng.choice([64, 128, 256, 512, 32 * rng.randint(1, 8)]), call=call)


# ------------------------------------------------------------------ matrices
def _degrees(case):
    """The degree sequence of a case, before the seed shuffles it over the rows."""
    n = case["n"]
    rng = np.random.Generator(np.random.PCG64(n))
    if case["degrees"] == "poisson":
        return np.minimum(np.maximum(rng.poisson(case["mean"], n), 1), n).astype(np.int64)
    if case["degrees"] == "powerlaw":
        return np.clip(rng.zipf(2.1, n), 1, min(13_000, n // 4)).astype(np.int64)
    return np.clip(np.rint(rng.lognormal(5.5, 1.2, n)), 1, min(21_000, n // 4)).astype(np.int64)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, *shape, lo=-1.0, hi=1.0, dtype=torch.float32):
    return (torch.rand(*shape, device="cuda", generator=g) * (hi - lo) + lo).to(dtype)


def _pointers(deg):
    out = torch.zeros(len(deg) + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(deg, 0, out=out[1:])
    return out


def _csr(case, g):
    """Square matrix with distinct sorted columns in every row: uniform ones, or (power-law graphs)
    columns whose popularity follows what preferential attachment over a fixed set of nodes gives."""
    n = case["n"]
    deg = torch.from_numpy(_degrees(case)).cuda()[torch.randperm(n, device="cuda", generator=g)]
    ptr = _pointers(deg)
    nnz = int(ptr[-1])
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    if case["degrees"] != "powerlaw":
        span = (n - deg + 1)[rows]
        cols = (torch.rand(nnz, device="cuda", generator=g, dtype=torch.float64) * span).long()
        cols = torch.minimum(cols, span - 1)
        del span
        key, _ = torch.sort(rows * (n + 1) + cols)
        cols = key - rows * (n + 1) + torch.arange(nnz, device="cuda") - ptr[:-1][rows]
    else:
        popular = torch.cumsum(torch.empty(n, device="cuda", dtype=torch.float64).exponential_(generator=g), 0)

        def some(k):
            at = torch.rand(k, device="cuda", generator=g, dtype=torch.float64) * popular[-1]
            return torch.searchsorted(popular, at).clamp_(max=n - 1)

        key, _ = torch.sort(rows * n + some(nnz))
        for _ in range(200):
            again = torch.zeros(nnz, dtype=torch.bool, device="cuda")
            again[1:] = key[1:] == key[:-1]
            k = int(again.sum())
            if k == 0:
                break
            key[again] = key[again] // n * n + some(k)
            key, _ = torch.sort(key)
        cols = key - rows * n
    return ptr.int(), cols.int(), deg, rows


def _buckets(case, ptr, cols, values):
    """The hyb decomposition on the device: (values, row ids, column ids) of every bucket."""
    n = case["n"]
    r, c, _, v, _ = fmt.column_part_hyb(n, n, ptr.cpu().numpy(), cols.cpu().numpy(), case["parts"], HYB_WIDTHS,
                                        data=values.cpu().numpy())
    up = lambda a: torch.from_numpy(a.reshape(-1)).cuda()  # noqa: E731
    return [(up(v[p][b]), up(r[p][b]), up(c[p][b])) for p in range(case["parts"]) for b in range(len(HYB_WIDTHS))
            if len(r[p][b])]


def _relation_edges(case):
    """Edges of every relation: Zipf(1.5) shares, at least one."""
    share = np.arange(1, case["rels"] + 1, dtype=np.float64) ** -1.5
    counts = np.maximum(np.floor(share / share.sum() * case["edges"]).astype(np.int64), 1)
    counts[0] += case["edges"] - counts.sum()
    return counts


def _csf(case, g):
    """Relation-major CSF of uniformly drawn edges: level-0 pointers and rows, level-1 pointers and
    columns, and how many entries every (relation, row) pair has."""
    n = case["n"]
    counts = torch.from_numpy(_relation_edges(case)).cuda()
    rel = torch.repeat_interleave(torch.arange(case["rels"], device="cuda"), counts)
    dst = torch.randint(0, n, (case["edges"],), device="cuda", generator=g)
    src = torch.randint(0, n, (case["edges"],), device="cuda", generator=g)
    key, _ = torch.sort((rel * n + dst) * n + src)
    pair, deg = torch.unique_consecutive(key // n, return_counts=True)
    ptr_i = torch.searchsorted(pair, torch.arange(case["rels"] + 1, device="cuda") * n)
    return ptr_i.int(), (pair % n).int(), _pointers(deg).int(), (key % n).int(), deg


def _pairs_in(case):
    """Expected number of (relation, row) pairs that have an edge."""
    n = case["n"]
    return float(np.sum(n * -np.expm1(_relation_edges(case) * math.log1p(-1.0 / n))))


# ------------------------------------------------------------------ what a program has in hand
def prepare(case, seed):
    g = _generator(seed)
    state = {"op": case["op"], "call": case.get("call")}
    PREPARE[case["op"]](case, g, state)
    if case.get("call") == "kept":
        state["kept"] = state["f"].prepare(*state["args"]())
    return state


def _prepare_csr_spmm(case, g, s):
    n, feat = case["n"], case["feat"]
    ptr, cols, deg, rows = _csr(case, g)
    a = (1.0 / deg.float())[rows]
    x, y = _uniform(g, n * feat), torch.zeros(n * feat, device="cuda")
    s.update(f=ops.csrmm, out=y, args=lambda: (a, x, y, ptr, cols))


def _prepare_hyb_spmm(case, g, s):
    n, feat = case["n"], case["feat"]
    ptr, cols, deg, rows = _csr(case, g)
    buckets = _buckets(case, ptr, cols, (1.0 / deg.float())[rows])
    x, y = _uniform(g, n, feat), torch.zeros(n, feat, device="cuda")
    # with one column partition every output row is written; with several everything is added to
    # a result that the call clears
    flags = 0 if case["parts"] == 1 else ops.L.HYB_ALL_ATOMIC | ops.L.HYB_ZERO_C
    s.update(f=ops.hyb_spmm, out=y, args=lambda: ops.hyb_args(x, y, buckets, feat, flags))


def _prepare_sddmm(case, g, s):
    n, feat = case["n"], case["feat"]
    ptr, cols, _, _ = _csr(case, g)
    scale, out = _uniform(g, len(cols), lo=0.0), torch.empty(len(cols), device="cuda")
    a, b = _uniform(g, n * feat), _uniform(g, n * feat)
    s.update(f=ops.sddmm, out=out, args=lambda: (a, b, out, ptr, cols, scale))


def _blocks(case):
    """Stored blocks of every block row: the diagonal and a fixed share of the others."""
    nb = case["n"] // case["blk"]
    rng = np.random.Generator(np.random.PCG64(case["n"]))
    return 1 + rng.binomial(nb - 1, case["density"], nb).astype(np.int64)


def _prepare_bsrmm(case, g, s):
    blk, feat = case["blk"], case["feat"]
    nb = case["n"] // blk
    deg = torch.from_numpy(_blocks(case)).cuda()
    order = torch.rand(nb, nb, device="cuda", generator=g)
    order.fill_diagonal_(-1.0)
    rank = torch.argsort(torch.argsort(order, 1), 1)
    at = torch.nonzero(rank < deg[:, None])
    ptr, cols = _pointers(deg).int(), at[:, 1].int().contiguous()
    nnzb = len(cols)
    a = torch.randn(nnzb * blk * blk, device="cuda", generator=g).half()
    b = torch.randn(nb * blk * feat, device="cuda", generator=g).half()
    c = torch.zeros(nb * blk * feat, device="cuda")
    s.update(f=ops.bsrmm, out=c, args=lambda: (a, b, c, ptr, cols, nb, nb, nnzb, blk, feat))


def _prepare_rgms(case, g, s):
    n, feat = case["n"], case["feat"]
    ptr_i, rows, ptr_j, cols, deg = _csf(case, g)
    a = torch.repeat_interleave(1.0 / deg.float(), deg)
    w = torch.randn(case["rels"] * feat * feat, device="cuda", generator=g) / math.sqrt(feat)
    x, y = _uniform(g, n * feat), torch.zeros(n * feat, device="cuda")
    s.update(f=ops.rgms, out=y, adds=True, args=lambda: (a, w, x, y, ptr_i, rows, ptr_j, cols))


def _prepare_rgcn_f16(case, g, s):
    n, fi, fo = case["n"], case["feat_in"], case["feat_out"]
    widths = [1, 2, 4, 8, 16, 32]
    ptr_i, rows, ptr_j, cols, _ = _csf(case, g)
    ip, r, c, m = fmt.csf_to_ell3d(*(t.cpu().numpy() for t in (ptr_i, rows, ptr_j, cols)), [32 // k for k in widths], widths)
    up = lambda t: torch.from_numpy(t).cuda()  # noqa: E731
    buckets = []
    for b in range(len(widths)):
        if len(r[b]) == 0:
            continue
        mask = up(m[b]).float()
        mid = up(np.repeat(np.arange(case["rels"], dtype=np.int32), np.diff(ip[b])))
        buckets.append(((mask / mask.sum(-1, keepdim=True).clamp_(min=1.0)).half(), up(r[b]), up(c[b]), mid))
    w = (torch.randn(case["rels"] * fi * fo, device="cuda", generator=g) / math.sqrt(fi)).half()
    x, y = _uniform(g, n * fi, dtype=torch.float16), torch.zeros(n * fo, device="cuda")
    s.update(f=ops.rgms_ell3d_f16, out=y, adds=True, args=lambda: ops.rgms_ell3d_f16_args(w, x, y, buckets, fi, fo))


def _conv_pairs(case):
    """(input, output) pairs of every kernel offset: the centre maps every point to itself, the
    others a share of the points."""
    rng = np.random.Generator(np.random.PCG64(case["n"]))
    counts = rng.binomial(case["n"], case["fill"], case["offsets"]).astype(np.int64)
    counts[case["offsets"] // 2] = case["n"]
    return counts


def _prepare_sparse_conv(case, g, s):
    n, fi, fo = case["n"], case["feat_in"], case["feat_out"]
    counts, maps = _conv_pairs(case), []
    for k, size in enumerate(counts):
        outs = torch.sort(torch.randperm(n, device="cuda", generator=g)[:size])[0]
        ins = outs if k == case["offsets"] // 2 else torch.randint(0, n, (int(size),), device="cuda", generator=g)
        maps.append(torch.stack([ins, outs], 1))
    plan = SparseConvPlan(torch.cat(maps), counts, False, n, n)
    x = _uniform(g, n, fi, dtype=torch.float16)
    w = (torch.randn(case["offsets"], fi, fo, device="cuda", generator=g) / math.sqrt(fi * case["offsets"])).half()
    s.update(f=None, plan=plan, x=x, w=w)


def _prepare_fusedmm(case, g, s):
    n, feat = case["n"], case["feat"]
    ptr, cols, _, _ = _csr(case, g)
    q = _uniform(g, n * feat) * (2.0 / math.sqrt(feat))
    k, v, o = _uniform(g, n * feat), _uniform(g, n * feat), torch.empty(n * feat, device="cuda")
    s.update(f=ops.fusedmm, out=o, args=lambda: (q, k, v, o, ptr, cols))


def _prepare_tcspmm(case, g, s):
    n, feat, t = case["n"], case["feat"], 16
    ptr, cols, _, _ = _csr(case, g)
    gp, tiles, mask = fmt.condense(ptr.cpu().numpy(), cols.cpu().numpy(), t, t)
    mb, nb, groups = len(gp) - 1, -(-n // t), len(tiles)
    up = lambda x: torch.from_numpy(x.reshape(-1)).cuda()  # noqa: E731
    a, gp, tiles = up(mask).half(), up(gp), up(tiles)
    x = torch.zeros(nb * t * feat, device="cuda", dtype=torch.float16)
    x[:n * feat] = _uniform(g, n * feat, dtype=torch.float16)
    y = torch.empty(mb * t * feat, device="cuda", dtype=torch.float16)
    s.update(f=ops.tcspmm, out=y, args=lambda: (a, x, y, gp, tiles, mb, nb, groups, feat, t, t))


PREPARE = {"csr_spmm": _prepare_csr_spmm, "hyb_spmm": _prepare_hyb_spmm, "sddmm": _prepare_sddmm,
           "bsrmm": _prepare_bsrmm, "rgms": _prepare_rgms, "rgcn_f16": _prepare_rgcn_f16,
           "sparse_conv": _prepare_sparse_conv, "fusedmm": _prepare_fusedmm, "tcspmm": _prepare_tcspmm}


# ------------------------------------------------------------------ one pass
def run(state):
    if state["op"] == "sparse_conv":
        return state["plan"](state["x"], state["w"])
    if state.get("adds"):  # the operator adds to its output: clearing it is part of a layer
        state["out"].zero_()
    if state["call"] == "kept":
        state["kept"]()
    else:
        state["f"](*state["args"]())
    return state["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    op, n = case["op"], case["n"]
    if "degrees" in case:
        nnz, feat = int(_degrees(case).sum()), case["feat"]
        index = 4 * (n + 1) + 4 * nnz
        if op in ("csr_spmm", "hyb_spmm"):
            return {"bytes": index + 4 * nnz + 8 * n * feat, "flops": 2.0 * nnz * feat}
        if op == "sddmm":
            return {"bytes": index + 8 * nnz + 8 * n * feat, "flops": 2.0 * nnz * feat}
        if op == "fusedmm":
            return {"bytes": index + 16 * n * feat, "flops": 4.0 * nnz * feat}
        # a 0/1 matrix with fp16 operands: its pattern, the operand and the result
        return {"bytes": index + 4 * n * feat, "flops": 2.0 * nnz * feat}
    if op == "bsrmm":
        blk, feat, nnzb = case["blk"], case["feat"], int(_blocks(case).sum())
        return {"bytes": 2 * nnzb * blk * blk + 4 * nnzb + 4 * (n // blk + 1) + 6 * n * feat,
                "flops": 2.0 * nnzb * blk * blk * feat}
    if op == "rgms":
        feat, pairs = case["feat"], _pairs_in(case)
        return {"bytes": 8 * case["edges"] + 8 * pairs + 4 * case["rels"] * feat * feat + 8 * n * feat,
                "flops": 2.0 * case["edges"] * feat + 2.0 * pairs * feat * feat}
    fi, fo = case["feat_in"], case["feat_out"]
    if op == "rgcn_f16":
        pairs = _pairs_in(case)
        return {"bytes": 6 * case["edges"] + 8 * pairs + 2 * case["rels"] * fi * fo + 2 * n * fi + 4 * n * fo,
                "flops": 2.0 * case["edges"] * fi + 2.0 * pairs * fi * fo}
    pairs = int(_conv_pairs(case).sum())
    return {"bytes": 8 * pairs + 2 * case["offsets"] * fi * fo + 2 * n * fi + 2 * n * fo, "flops": 2.0 * pairs * fi * fo}


def tolerance(case):
    if case["op"] in ("rgcn_f16", "sparse_conv", "tcspmm"):
        return {"rel": 2e-3}  # fp16 intermediates or results
    if case["op"] == "fusedmm":
        return {"rel": 2e-5}  # three fp32 stages, the second an exponential
    return {"rel": 1e-5}      # fp32 sums
