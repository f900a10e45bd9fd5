"""``SO3Linear`` on straight-line Clebsch-Gordan blocks: 'uu' in one kernel per direction, the channel-wise half of
'uv' (operator layer over ``eqt_so3_uu_*`` / ``eqt_so3_uv_*``)."""
from __future__ import annotations

import ctypes as C
from typing import Optional, Sequence, Tuple

import numpy as np
import torch
from torch import Tensor

from .. import _lib
from ..csrc.gen_path_specs import MAX_L as PATH_MAX_L

_PATH = np.dtype([("code", "<i4"), ("offset", "<i4"), ("offset_y", "<i4"), ("weight", "<i4"), ("scale", "<f4"),
                  ("row", "<i4"), ("row_stride", "<i4")])
_BLOCK = np.dtype([("l", "<i4"), ("offset", "<i4"), ("first", "<i4"), ("count", "<i4")])


class PathPlan:
    """Device tables of one layer for the one-pass kernels.  ``paths``: (k, i, j) of every weight - output, first and
    second operand irrep - and ``scales`` the factors on their Clebsch-Gordan blocks."""

    def __init__(self, paths: Sequence[Tuple[int, int, int]], scales: Sequence[float], irreps_out, irreps1, irreps2, device):
        self.device, self._fits, self.mix = torch.device(device), {}, None      # mix: tables of the weight step ('uv'), False: other rows
        ls = [[ir.l for ir in irs] for irs in (irreps_out, irreps1, irreps2)]
        # a path of degrees that do not couple has no block (its entries in the layer's tables are none either)
        self.usable = (len(paths) > 0 and all(0 <= l <= PATH_MAX_L for degrees in ls for l in degrees)
                       and all(abs(ls[1][i] - ls[2][j]) <= ls[0][k] <= ls[1][i] + ls[2][j] for k, i, j in paths))
        if not self.usable:
            return
        start = [np.cumsum([0] + [2 * l + 1 for l in degrees]).tolist() for degrees in ls]
        # rows of the intermediate: per output irrep, component by component, its paths ordered by (i, j, weight)
        row, fan, num_rows, self.row_weights = {}, {}, 0, []
        for k, l in enumerate(ls[0]):
            mine = sorted((w for w in range(len(paths)) if paths[w][0] == k), key=lambda w: (paths[w][1], paths[w][2], w))
            self.row_weights += [mine] * (2 * l + 1)              # of every output component
            row.update((w, num_rows + n) for n, w in enumerate(mine))
            fan[k] = len(mine)
            num_rows += len(mine) * (2 * l + 1)
        parts = []
        for key, other in ((0, 1), (1, 0)):
            order = sorted(range(len(paths)), key=lambda w: paths[w][key])
            parts.append(np.array([(4 * ls[other][paths[w][other]] + ls[2][paths[w][2]], start[other][paths[w][other]],
                                    start[2][paths[w][2]], w, scales[w], row[w], fan[paths[w][0]]) for w in order], dtype=_PATH))
            first = np.searchsorted([paths[w][key] for w in order], np.arange(len(ls[key]) + 1)).tolist()
            parts.append(np.array([(l, start[key][n], first[n], first[n + 1] - first[n]) for n, l in enumerate(ls[key])], dtype=_BLOCK))
        parts.append(np.array([row[w] + m * fan[paths[w][0]] for w in order for m in range(2 * ls[0][paths[w][0]] + 1)], dtype=np.int32))
        # one upload: the parts back to back, each on a 16-byte boundary
        blob, at, size = [], [], 0
        for part in parts:
            at.append(size)
            raw = part.tobytes()
            blob.append(raw + b"\0" * (-len(raw) % 16))
            size += len(blob[-1])
        self.blob = torch.frombuffer(bytearray(b"".join(blob)), dtype=torch.uint8).to(device)
        base = self.blob.data_ptr()
        self.sizes = (start[1][-1], start[2][-1], start[0][-1], len(paths))
        self.num_rows = num_rows
        self.struct = _lib.PathTableStruct(base + at[1], base + at[3], base + at[0], base + at[2], base + at[4], *self.sizes,
                                           len(paths), len(ls[0]), len(ls[1]), num_rows)
        self.ref = C.byref(self.struct)

    def rows_match(self, info) -> bool:
        """Whether the rows of the intermediate that ``info`` (the forward table of the weight step) consumes are the rows
        of this plan.  They are not where a path is listed twice: the table then has a row per run of a weight among the
        entries of a component, several for one (component, weight)."""
        if not self.usable or info.index1 is not None or info.scale is not None or info.gather_index is not None \
                or info.index_out is not None or info.out_size != len(self.row_weights):
            return False
        seg = list(range(info.out_size + 1)) if info.seg_out is None else info.seg_out.tolist()
        weights = list(range(seg[-1])) if info.index2 is None else info.index2.tolist()
        return len(weights) == self.num_rows and [weights[a:b] for a, b in zip(seg, seg[1:])] == self.row_weights

    def supported(self, x: Tensor, y: Tensor, w: Tensor) -> bool:
        if not (self.usable and x.is_cuda and x.dtype in (torch.float32, torch.bfloat16) and x.dtype == y.dtype == w.dtype
                and x.ndim == 3 and y.ndim == 2 and x.shape[0] == y.shape[0] and x.shape[0] > 0 and w.ndim in (2, 3)
                and x.shape[2] == w.shape[-1] and x.shape[1] == self.sizes[0] and y.shape[1] == self.sizes[1]
                and w.shape[-2] == self.sizes[3] and (w.ndim == 2 or w.shape[0] == x.shape[0])
                and y.device == x.device == w.device == self.device):
            return False
        key = (x.shape[2], w.ndim, x.dtype)
        if key not in self._fits:
            self._fits[key] = all(_lib.lib().eqt_so3_uu_scratch_floats(self.ref, n, x.shape[2], int(w.ndim == 3),
                                                                       _lib.DTYPE_CODE[x.dtype]) >= 0 for n in (1, 1 << 30))
        return self._fits[key] and (x.data_ptr() | w.data_ptr()) % 16 == 0

    def uv_supported(self, x: Tensor, y: Tensor, w: Tensor) -> bool:
        """Whether the channel-wise kernels of the 'uv' layer take these operands (float32, weights shared by the batch)."""
        if not (self.usable and x.is_cuda and x.dtype == torch.float32 and x.dtype == y.dtype == w.dtype
                and x.ndim == 3 and y.ndim == 2 and x.shape[0] == y.shape[0] and x.shape[0] > 0 and w.ndim == 3
                and x.shape[2] == w.shape[1] and x.shape[1] == self.sizes[0] and y.shape[1] == self.sizes[1]
                and w.shape[0] == self.sizes[3] and y.device == x.device == w.device == self.device):
            return False
        key = ("uv", x.shape[2])
        if key not in self._fits:
            self._fits[key] = bool(_lib.lib().eqt_so3_uv_supported(self.ref, x.shape[2]))
        return self._fits[key] and (x.data_ptr() | w.data_ptr()) % 16 == 0


def so3_uv_expand(plan: PathPlan, x: Tensor, y: Tensor) -> Tensor:
    """``rows[n, r, c]``: the entries of (output component, path) row r contracted with x and y; contiguous float32."""
    n, _, c = x.shape
    rows = torch.empty(n, plan.num_rows, c, dtype=torch.float32, device=x.device)
    with _lib.on_device(x.device):
        _lib.check(_lib.lib().eqt_so3_uv_expand(plan.ref, x.data_ptr(), y.data_ptr(), rows.data_ptr(), n, c, _lib.stream_ptr(x.device)),
                   "eqt_so3_uv_expand")
    return rows


def aligned(*tensors: Optional[Tensor]) -> bool:
    return all(t is None or t.data_ptr() % 16 == 0 for t in tensors)


def so3_uv_backward(plan: PathPlan, x: Optional[Tensor], y: Optional[Tensor], grad_rows: Tensor,
                    need: Tuple[bool, bool]) -> Tuple[Optional[Tensor], Optional[Tensor]]:
    """Gradients of :func:`so3_uv_expand` with respect to x and y, from one pass over ``grad_rows``; the gradient of x takes
    y and that of y takes x."""
    n, _, c = grad_rows.shape
    gx = grad_rows.new_empty(n, plan.sizes[0], c) if need[0] else None
    gy = grad_rows.new_empty(n, plan.sizes[1]) if need[1] else None
    dev = grad_rows.device
    with _lib.on_device(dev):
        _lib.check(_lib.lib().eqt_so3_uv_backward(plan.ref, _lib.ptr(x), _lib.ptr(y), grad_rows.data_ptr(), _lib.ptr(gx), _lib.ptr(gy),
                                                  n, c, _lib.stream_ptr(dev)), "eqt_so3_uv_backward")
    return gx, gy


def so3_uu_forward(plan: PathPlan, x: Tensor, y: Tensor, w: Tensor) -> Tensor:
    """``out[n, M, c] = sum_t s_t x[n, M1_t, c] y[n, M2_t] w[(n,) p_t, c]``; contiguous operands of one dtype."""
    n, _, c = x.shape
    out = torch.empty(n, plan.sizes[2], c, dtype=x.dtype, device=x.device)
    with _lib.on_device(x.device):
        _lib.check(_lib.lib().eqt_so3_uu_forward(plan.ref, x.data_ptr(), y.data_ptr(), w.data_ptr(), out.data_ptr(), n, c,
                                                 int(w.ndim == 3), _lib.DTYPE_CODE[x.dtype], _lib.stream_ptr(x.device)),
                   "eqt_so3_uu_forward")
    return out


def so3_uu_backward(plan: PathPlan, x: Optional[Tensor], y: Optional[Tensor], w: Optional[Tensor], g: Tensor, need: Tuple[bool, bool, bool],
                    per_sample: bool) -> Tuple[Optional[Tensor], Optional[Tensor], Optional[Tensor]]:
    """Gradients with respect to x, y and w (``None`` where not needed), all from one launch; each takes the other two."""
    n, _, c = g.shape
    d1, d2, _, p = plan.sizes
    shapes = ((n, d1, c), (n, d2), (n, p, c) if per_sample else (p, c))
    gx, gy, gw = (g.new_empty(shape) if wanted else None for shape, wanted in zip(shapes, need))
    lib, scratch, floats, dev = _lib.lib(), None, 0, g.device
    with _lib.on_device(dev):
        if need[2] and not per_sample:
            floats = int(lib.eqt_so3_uu_scratch_floats(plan.ref, n, c, 0, _lib.DTYPE_CODE[g.dtype]))
            scratch = torch.empty(floats, dtype=torch.float32, device=dev)
        _lib.check(lib.eqt_so3_uu_backward(plan.ref, _lib.ptr(x), _lib.ptr(y), _lib.ptr(w), g.data_ptr(), _lib.ptr(gx), _lib.ptr(gy),
                                           _lib.ptr(gw), _lib.ptr(scratch), floats, n, c, int(per_sample), _lib.DTYPE_CODE[g.dtype],
                                           _lib.stream_ptr(dev)), "eqt_so3_uu_backward")
    return gx, gy, gw
