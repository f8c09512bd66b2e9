"""Sparse convolution through the RGMS operator: the caller side of
examples/rgms/sparse_conv/sparse_conv.py:93-125 of the reference.

A sparse (submanifold / strided / transposed) convolution layer arrives the way torchsparse
hands it over: ``inputs [n_in, feat_in]``, ``weights [K, feat_in, feat_out]`` (one matrix per
kernel offset), ``nbmaps [pairs, 2]`` listing (input point, output point) pairs grouped by kernel
offset, ``nbsizes [K]`` the number of pairs of every offset, and ``transposed`` (the maps of a
transposed convolution are stored the other way round).  The layer computes

    y[o] = sum over offsets k, pairs (i, o) of offset k:  x[i] @ weights[k]

The reference turns the maps into a heterogeneous graph with one relation per kernel offset
(sparse_conv.py:93-104), that graph into a 3-level CSF tensor in which EVERY output point is a
level-0 row of EVERY relation (examples/rgms/sparse_conv/rgms.py:677-692), the CSF tensor into
ELL3D buckets with ``buckets = [1]`` and groups of ``ty * 16 = 128`` rows (rgms.py:701-710), and
calls the tensor-core RGMS function with ``W`` as ``[K, feat_in, feat_out]`` (the two
``transpose(-1, -2)`` of sparse_conv.py:113 and rgms.py:842 cancel).  The same steps here, with the
library's ``csf_to_ell3d`` and ``sparsetir_rgms_ell3d_f16``.
"""
from __future__ import annotations

from typing import List, Optional, Sequence, Tuple

import numpy as np
import torch

from . import format as fmt
from . import ops


def relations_from_maps(nbmaps, nbsizes, transposed: bool) -> List[Tuple[np.ndarray, np.ndarray]]:
    """(sources, destinations) of every kernel offset, as sparse_conv.py:96-103 slices them:
    offset ``rel`` owns ``nbsizes[rel]`` consecutive rows of ``nbmaps``; column 0 is the input
    point and column 1 the output point, swapped for a transposed convolution."""
    maps = np.asarray(nbmaps.cpu() if isinstance(nbmaps, torch.Tensor) else nbmaps)
    sizes = [int(s) for s in (nbsizes.tolist() if hasattr(nbsizes, "tolist") else nbsizes)]
    if maps.ndim != 2 or maps.shape[1] != 2:
        raise ValueError("nbmaps must have shape [pairs, 2]")
    if sum(sizes) > maps.shape[0]:
        raise ValueError("nbsizes counts more pairs than nbmaps holds")
    out, offset = [], 0
    for size in sizes:
        i = maps[offset:offset + size, 0]
        o = maps[offset:offset + size, 1]
        offset += size
        if transposed:
            i, o = o, i
        out.append((np.asarray(i, np.int64), np.asarray(o, np.int64)))
    return out


def csf_from_relations(rels: Sequence[Tuple[np.ndarray, np.ndarray]], num_dst: int):
    """The CSF arrays rgms.py:677-697 builds from the graph: per relation the CSC of its
    (destination x source) adjacency over ALL ``num_dst`` destinations, so
    ``indptr_0 = [0, m, 2m, ...]`` and ``indices_0 = arange(m)`` repeated; level 1 lists the
    sources of every destination (pairs of one destination keep their order in the maps)."""
    m = int(num_dst)
    indptr_0 = (np.arange(len(rels) + 1, dtype=np.int64) * m)
    indices_0 = np.tile(np.arange(m, dtype=np.int32), len(rels))
    ptr_parts, idx_parts, base = [np.zeros(1, np.int64)], [], 0
    for src, dst in rels:
        order = np.argsort(dst, kind="stable")
        counts = np.bincount(dst, minlength=m)
        if len(counts) > m:
            raise ValueError("an output index exceeds the number of output points")
        ptr_parts.append(base + np.cumsum(counts))
        idx_parts.append(src[order].astype(np.int32))
        base += len(src)
    indptr_1 = np.concatenate(ptr_parts)
    indices_1 = np.concatenate(idx_parts) if idx_parts else np.zeros(0, np.int32)
    if indptr_0[-1] > np.iinfo(np.int32).max or base > np.iinfo(np.int32).max:
        raise ValueError("the layer is too large for 32-bit indices")
    return indptr_0.astype(np.int32), indices_0, indptr_1.astype(np.int32), indices_1


def ell3d_from_maps(nbmaps, nbsizes, transposed: bool, num_inputs: int,
                    num_outputs: Optional[int] = None, group_size: int = 128,
                    buckets: Sequence[int] = (1,)):
    """Host side of the conversion: ``(buckets, num_outputs, num_pairs)`` with one
    ``(a float16, rows, cols, mid)`` tuple of numpy arrays per ELL3D bucket — the arrays the
    reference passes to the built function (rgms.py:846-855): the 0/1 mask as values, the row and
    column ids of CSFToELL3D, and the relation of every group."""
    rels = relations_from_maps(nbmaps, nbsizes, bool(transposed))
    top_dst = max((int(d.max()) for _, d in rels if len(d)), default=-1)
    top_src = max((int(s.max()) for s, _ in rels if len(s)), default=-1)
    m = int(num_outputs) if num_outputs is not None else top_dst + 1
    if top_dst >= m or top_src >= int(num_inputs):
        raise ValueError("nbmaps names a point beyond the given number of points")
    if any(len(d) and (int(d.min()) < 0 or int(s.min()) < 0) for s, d in rels):
        raise ValueError("nbmaps holds a negative index")
    buckets = [int(b) for b in buckets]
    ip0, ix0, ip1, ix1 = csf_from_relations(rels, m)
    indptr, rows, cols, mask = fmt.csf_to_ell3d(ip0, ix0, ip1, ix1,
                                                [group_size // b for b in buckets], buckets)
    out = []
    for b in range(len(buckets)):
        mid = np.repeat(np.arange(len(rels), dtype=np.int32), np.diff(indptr[b]))
        out.append((mask[b].astype(np.float16), rows[b], cols[b], mid))
    return out, m, int(sum(len(s) for s, _ in rels))


def neighbour_map(nbmaps, nbsizes, transposed: bool, num_outputs: int, device: torch.device) -> Optional[torch.Tensor]:
    """The layer's pairs as ``sparsetir_sparse_conv_f16`` takes them, on ``device``: tiles of 128 outputs,
    ``map[(tile * K + k) * 128 + t]`` = input point of output ``tile * 128 + t`` at kernel offset ``k``,
    or -1; None when an (offset, output) pair repeats."""
    maps = nbmaps if isinstance(nbmaps, torch.Tensor) else torch.from_numpy(np.array(nbmaps, dtype=np.int64))
    maps = maps.to(device, torch.int64)
    sizes = torch.as_tensor([int(s) for s in (nbsizes.tolist() if hasattr(nbsizes, "tolist") else nbsizes)],
                            dtype=torch.int64).to(device)
    offsets, pairs = len(sizes), int(sizes.sum())
    src, dst = (maps[:pairs, 1], maps[:pairs, 0]) if transposed else (maps[:pairs, 0], maps[:pairs, 1])
    rel = torch.repeat_interleave(torch.arange(offsets, device=device), sizes, output_size=pairs)
    out = torch.full((-(-num_outputs // 128) * offsets * 128,), -1, dtype=torch.int32, device=device)
    out[(dst // 128 * offsets + rel) * 128 + dst % 128] = src.int()
    return out if int((out >= 0).sum()) == pairs else None


def map_pays(num_outputs: int, offsets: int, pairs: int, feat_in: int, feat_out: int) -> bool:
    """Whether the kernel over the neighbour map is the faster one for these sizes.

    It multiplies the full ``128 x (offsets * feat_in)`` operand of every tile whatever the share of
    pairs; the buckets' tensor-core kernel pays per pair, but takes only multiples of 64 channels and
    builds a map of its own on every call when ``feat_out >= 2 * feat_in``.  Measured on 4,000 to
    100,000 points, 8 and 27 offsets, 20 to 60 % of the pairs (float16 result, us, map / buckets):
    100,000 x 27, 64 -> 64 channels 41 / 39 at 20 %, 41 / 53 at 35 %, 41 / 79 at 60 %; 128 -> 64 76 / 66 at 35 %,
    76 / 99 at 60 %; 30,000 x 27, 128 -> 128 33 / 29 at 20 %, 33 / 37 at 35 %, 256 -> 256 80 / 72 at 35 %, 82 / 103
    at 60 %; 4,000 x 8 12 / 22.  The two estimates follow these within about 20 %, and where they choose the slower
    one it is so by 10 % at most."""
    if feat_in % 16 != 0 or feat_out % 32 != 0 or not 0 < feat_out <= 256 or feat_in <= 0:
        return False
    if feat_in % 64 != 0 or feat_out % 64 != 0 or feat_out >= 2 * feat_in:
        return True
    waves = -(-num_outputs // (128 * 148))  # tiles of 128 outputs on 148 SMs
    by_map = 6.0 + waves * offsets * feat_in / 64 * (0.40 if feat_out > 128 else 0.27 if feat_out > 64 else 0.22)
    by_pairs = max(24.0, 18.0 + pairs * 1e-6 * (0.30 * feat_in + 0.34 * feat_out - 4.0))
    return by_map <= by_pairs


class SparseConvPlan:
    """The structure of one layer, converted once (host side) and kept on the device.

    A layer whose (offset, output) pairs never repeat is kept as a neighbour map too: where
    ``map_pays`` says so a call is one launch of ``sparsetir_sparse_conv_f16``, which writes its
    result; all others run ``sparsetir_rgms_ell3d_f16`` on the ELL3D buckets.

    ``plan(inputs, weights)`` then runs the operator; the maps of a layer do not change between
    calls, so the host conversion is not part of the steady state (the reference also converts
    before it times, rgms.py:677-710 against :861-864)."""

    _map: Optional[torch.Tensor] = None  # also of a plan that was saved when plans had no map

    def __init__(self, nbmaps, nbsizes, transposed: bool, num_inputs: int,
                 num_outputs: Optional[int] = None, device: Optional[torch.device] = None,
                 group_size: int = 128, buckets: Sequence[int] = (1,)):
        host, self.num_outputs, self.num_pairs = ell3d_from_maps(
            nbmaps, nbsizes, transposed, num_inputs, num_outputs, group_size, buckets)
        self.num_inputs = int(num_inputs)
        self.num_offsets = len(nbsizes)
        self.device = device if device is not None else torch.device("cuda", torch.cuda.current_device())
        self.buckets = [tuple(torch.from_numpy(np.ascontiguousarray(a)).to(self.device) for a in bk)
                        for bk in host]
        # at most 1 GB: layers beyond that, and layers with repeated pairs, keep the buckets alone
        if self.num_pairs > 0 and self.num_offsets * self.num_outputs <= 1 << 28:
            self._map = neighbour_map(nbmaps, nbsizes, bool(transposed), self.num_outputs, self.device)

    def __call__(self, inputs: torch.Tensor, weights: torch.Tensor,
                 out: Optional[torch.Tensor] = None, out_dtype: torch.dtype = torch.float16) -> torch.Tensor:
        if inputs.dim() != 2 or weights.dim() != 3:
            raise ValueError("inputs must be [n_in, feat_in] and weights [K, feat_in, feat_out]")
        if inputs.shape[0] != self.num_inputs or weights.shape[0] != self.num_offsets:
            raise ValueError("inputs / weights do not match the layer this plan was made for")
        feat_in, feat_out = int(weights.shape[1]), int(weights.shape[2])
        if inputs.shape[1] != feat_in:
            raise ValueError("inputs and weights disagree on feat_in")
        x = inputs.to(self.device, torch.float16).contiguous()
        w = weights.to(self.device, torch.float16).contiguous()
        mapped = (self._map is not None
                  and map_pays(self.num_outputs, self.num_offsets, self.num_pairs, feat_in, feat_out)
                  and (out_dtype if out is None else out.dtype) in (torch.float16, torch.float32)
                  and (x.data_ptr() | w.data_ptr() | (0 if out is None else out.data_ptr())) % 16 == 0)
        add = out is not None
        if out is None:
            make = torch.empty if mapped else torch.zeros
            out = make(self.num_outputs, feat_out, dtype=out_dtype, device=self.device)
        elif tuple(out.shape) != (self.num_outputs, feat_out) or not out.is_contiguous():
            raise ValueError("out must be a contiguous [num_outputs, feat_out] tensor (it is added to)")
        if mapped:
            ops.sparse_conv_f16(w.view(-1), x.view(-1), out.view(-1), self._map, self.num_outputs, self.num_offsets, feat_in,
                                feat_out, int(add))
            return out
        ops.rgms_ell3d_f16(*ops.rgms_ell3d_f16_args(w, x, out, self.buckets, feat_in, feat_out))
        return out


def sparse_conv(inputs: torch.Tensor, weights: torch.Tensor, nbmaps, nbsizes, transposed: bool = False,
                num_outputs: Optional[int] = None, out_dtype: torch.dtype = torch.float16) -> torch.Tensor:
    """One call with the reference driver's inputs (sparse_conv.py:52-61): ``y [n_out, feat_out]``,
    float16 like the reference's output unless ``out_dtype`` says float32."""
    plan = SparseConvPlan(nbmaps, nbsizes, transposed, int(inputs.shape[0]), num_outputs,
                          device=inputs.device if inputs.is_cuda else None)
    return plan(inputs, weights, out_dtype=out_dtype)
