"""Radius graph and fused edge features (operator layer over the ``eqt_radius_*`` entry points)."""
from __future__ import annotations

import ctypes as C
import math
from typing import NamedTuple, Optional

import torch
from torch import Tensor

from .. import _lib

CUTOFF_KINDS = {"polynomial": 0, "cosine": 1, "mollifier": 2}

#: neighbour lists of at most this many entries (256 MB) are kept between the search and the pass that writes the edges;
#: above it that pass searches again
MAX_LIST_ENTRIES = 1 << 26
_LIST_ROW = 512          # most candidates of one target


class CellList(NamedTuple):
    cell_start: Tensor       # (cells + 1,) int32 first place of every cell
    sorted: Tensor           # (N, 4) float32: x, y, z and index (its bits) of the points by cell
    point_cell: Tensor       # (N,) int32, -1 for a graph index out of range
    dims: "C.Array"
    cell_size: float

    def struct(self):
        """The struct of the searching entry points and what it points at."""
        index = self.sorted[:, 3].contiguous().view(torch.int32)
        return _lib.RadiusGridStruct(self.cell_start.data_ptr(), index.data_ptr(), self.point_cell.data_ptr(), self.cell_size,
                                     self.dims), index


def build_cell_list(pos: Tensor, r: float, batch: Optional[Tensor] = None) -> CellList:
    """Bin ``pos`` (N, 3) into cubic cells of side ``r`` (slightly more), one slab of cells per graph."""
    n = pos.shape[0]
    dev = pos.device
    cell_size = float(r) * (1.0 + 1e-5)
    lo, hi = torch.stack(torch.aminmax(pos, dim=0)).tolist()            # one host synchronisation
    dims = [max(1, int(math.floor((b - a) / cell_size)) + 1) for a, b in zip(lo, hi)]
    per_graph = dims[0] * dims[1] * dims[2]
    graphs = 1 if batch is None else max(0, int(batch.max()) + 1)
    if graphs * per_graph >= 2 ** 31:
        raise ValueError("cell grid too large; the positions are too spread out for this cutoff")
    cells = graphs * per_graph
    batch = None if batch is None else batch.long().contiguous()
    counts = torch.zeros(2 * cells + 1, dtype=torch.int32, device=dev)  # [starts, counts]
    cell_start, cell_count = counts[:cells + 1], counts[cells + 1:]
    point_cell, rank = torch.empty(2, n, dtype=torch.int32, device=dev)
    placed = torch.empty(n, 4, dtype=torch.float32, device=dev)
    c_dims = (C.c_int32 * 3)(*dims)
    lib = _lib.lib()
    with _lib.on_device(dev):
        _lib.check(lib.eqt_radius_bin(pos.data_ptr(), _lib.ptr(batch), n, (C.c_float * 3)(*lo), cell_size, c_dims, graphs,
                                      point_cell.data_ptr(), rank.data_ptr(), cell_count.data_ptr(), _lib.stream_ptr(dev)),
                   "eqt_radius_bin")
        torch.cumsum(cell_count, 0, dtype=torch.int32, out=cell_start[1:])
        _lib.check(lib.eqt_radius_place(pos.data_ptr(), point_cell.data_ptr(), rank.data_ptr(), cell_start.data_ptr(),
                                        placed.data_ptr(), n, _lib.stream_ptr(dev)), "eqt_radius_place")
    return CellList(cell_start, placed, point_cell, c_dims, cell_size)


class EdgeFeatures(NamedTuple):
    src: Tensor                       # (E,) int64, ascending within a target
    dst: Tensor                       # (E,) int64, ascending
    ptr: Tensor                       # (N + 1,) int64 CSR by target
    vec: Optional[Tensor]             # (E, 3) pos[dst] - pos[src]
    length: Optional[Tensor]          # (E,)
    sh: Optional[Tensor]              # (E, (l_max + 1)^2)
    bessel: Optional[Tensor]          # (E, num_basis)
    cutoff: Optional[Tensor]          # (E,)


def radius_graph_features(pos: Tensor, r: float, batch: Optional[Tensor] = None, loop: bool = False,
                          max_num_neighbors: int = 32, with_vec: bool = True, with_length: bool = False,
                          l_max: Optional[int] = None, integral_normalize: bool = False,
                          bessel_weights: Optional[Tensor] = None, bessel_r_max: Optional[float] = None,
                          cutoff: Optional[str] = None, cutoff_r_max: Optional[float] = None, cutoff_r_min: float = 0.0,
                          cutoff_p: float = 6.0, cutoff_eps: float = 1e-7) -> EdgeFeatures:
    """Edges ``j -> i`` for ``|pos_i - pos_j| < r`` (same graph, at most ``max_num_neighbors`` per target, those of
    smallest index) sorted by (target, source), and the requested per-edge features, in two kernel passes."""
    dev = _lib.require_cuda(pos, batch, bessel_weights)
    if pos.dtype != torch.float32 or pos.ndim != 2 or pos.shape[1] != 3:
        raise TypeError("pos must be a float32 (N, 3) tensor")
    pos = pos.detach().contiguous()
    n = pos.shape[0]
    if n == 0:
        z = torch.zeros(0, dtype=torch.long, device=dev)
        return EdgeFeatures(z, z, torch.zeros(1, dtype=torch.long, device=dev), None, None, None, None, None)
    if l_max is not None and not 0 <= l_max <= 4:
        raise ValueError("the fused kernel takes l_max <= 4; use SphericalHarmonics on edge_vec for higher degrees")
    cells = build_cell_list(pos, r, batch)
    degree = torch.empty(n, dtype=torch.int32, device=dev)
    tail = torch.zeros(n + 2, dtype=torch.long, device=dev)              # CSR pointer, then the status of the search
    ptr, flag = tail[:n + 1], tail[n + 1:].view(torch.int32)
    row = min(int(max_num_neighbors), _LIST_ROW)
    lists = torch.empty(n, row, dtype=torch.int32, device=dev) if 0 < row and n * row <= MAX_LIST_ENTRIES else None
    lib = _lib.lib()
    with _lib.on_device(dev):
        if lists is not None:
            _lib.check(lib.eqt_radius_search(pos.data_ptr(), cells.sorted.data_ptr(), cells.cell_start.data_ptr(),
                                             cells.point_cell.data_ptr(), n, cells.dims, float(r), int(loop), row,
                                             degree.data_ptr(), lists.data_ptr(), flag.data_ptr(), _lib.stream_ptr(dev)),
                       "eqt_radius_search")
        else:
            grid, index = cells.struct()
            _lib.check(lib.eqt_radius_count(C.byref(grid), pos.data_ptr(), None, n, float(r), int(loop), int(max_num_neighbors),
                                            degree.data_ptr(), flag.data_ptr(), _lib.stream_ptr(dev)), "eqt_radius_count")
    torch.cumsum(degree, 0, out=ptr[1:])
    e, failed = tail[n:].tolist()                                        # host synchronisation: the output size
    if failed:
        raise _lib.EqtError("a node has more than 512 candidate neighbours; lower the cutoff")
    src = torch.empty(e, dtype=torch.long, device=dev)
    dst = torch.empty(e, dtype=torch.long, device=dev)
    f32 = dict(dtype=torch.float32, device=dev)
    vec = torch.empty(e, 3, **f32) if with_vec else None
    length = torch.empty(e, **f32) if with_length else None
    sh = torch.empty(e, (l_max + 1) ** 2, **f32) if l_max is not None else None
    bw = None if bessel_weights is None else bessel_weights.detach().to(**f32).contiguous()
    bes = torch.empty(e, bw.numel(), **f32) if bw is not None else None
    cut = torch.empty(e, **f32) if cutoff is not None else None
    if bw is not None and bessel_r_max is None:
        raise ValueError("bessel_r_max is required with bessel_weights")
    if cutoff is not None and cutoff_r_max is None:
        raise ValueError("cutoff_r_max is required with cutoff")
    feats = _lib.EdgeFeaturesStruct(_lib.ptr(vec), _lib.ptr(length), _lib.ptr(sh), _lib.ptr(bes), _lib.ptr(cut), _lib.ptr(bw),
                                    l_max or 0, int(integral_normalize), 0 if bw is None else bw.numel(),
                                    CUTOFF_KINDS[cutoff] if cutoff is not None else 0, float(bessel_r_max or 1.0),
                                    float(cutoff_r_min), float(cutoff_r_max or 1.0), float(cutoff_p), float(cutoff_eps))
    with _lib.on_device(dev):
        if lists is not None:
            _lib.check(lib.eqt_radius_list_edges(pos.data_ptr(), n, ptr.data_ptr(), lists.data_ptr(), row, src.data_ptr(),
                                                 dst.data_ptr(), C.byref(feats), _lib.stream_ptr(dev)), "eqt_radius_list_edges")
        else:
            _lib.check(lib.eqt_radius_edges(C.byref(grid), pos.data_ptr(), None, n, float(r), int(loop), int(max_num_neighbors),
                                            ptr.data_ptr(), src.data_ptr(), dst.data_ptr(), C.byref(feats), flag.data_ptr(),
                                            _lib.stream_ptr(dev)), "eqt_radius_edges")
    return EdgeFeatures(src, dst, ptr, vec, length, sh, bes, cut)
