"""Product of two channelled operands with full channel mixing ('uvw') without its intermediate (operator layer over
``eqt_uvw_contract`` / ``eqt_uvw_wgrad``)."""
from __future__ import annotations

import ctypes as C
from typing import Optional, Sequence, Tuple

import numpy as np
import torch
from torch import Tensor

from .. import _lib
from ..constants import so3_clebsch_gordan
from ..csrc.gen_path_specs import TRIPLE_MAX_L
from .fused_tp_op import status_flag

_PATH = np.dtype([("l_o", "<i4"), ("l_s", "<i4"), ("l_f", "<i4"), ("offset_o", "<i4"), ("offset_s", "<i4"), ("offset_f", "<i4"),
                  ("weight", "<i4"), ("scale", "<f4")])
# operands of the layer (0 = output, 1 = first, 2 = second operand) in the places (out, s, f) of a role
FORWARD, GRAD_1, GRAD_2 = (0, 1, 2), (1, 2, 0), (2, 1, 0)
_TILE = 128              # samples of a CTA


def exchanged_scale(degrees: Sequence[int], role: Tuple[int, int, int]) -> float:
    """Ratio of the Clebsch-Gordan block of ``degrees`` (output, first, second operand), its axes in the order of ``role``, to the
    block of the degrees in that order: the two are multiples of one another."""
    ours = so3_clebsch_gordan(*degrees).transpose(role)
    block = so3_clebsch_gordan(*(degrees[a] for a in role))
    return float((ours * block).sum() / (block * block).sum())


class _Role:
    def __init__(self, role, paths, scales, degrees, start):
        o, s, f = role
        self.dims = tuple(start[a][-1] for a in (s, f, o))
        order = sorted(range(len(paths)), key=lambda w: (paths[w][f], paths[w][o], w))
        ls = [tuple(degrees[a][paths[w][a]] for a in (0, 1, 2)) for w in range(len(paths))]
        self.table = np.array([(ls[w][o], ls[w][s], ls[w][f], start[o][paths[w][o]], start[s][paths[w][s]], start[f][paths[w][f]], w,
                                scales[w] * exchanged_scale(ls[w], role)) for w in order], dtype=_PATH)
        self.degrees = (C.c_int32 * (3 * len(order)))(*(ls[w][a] for w in order for a in (o, s, f)))
        outs = [[paths[w][o] for w in order if paths[w][f] == n] for n in range(len(degrees[f]))]
        self.groups = (_lib.UvwGroupStruct * len(degrees[f]))(
            *(_lib.UvwGroupStruct(l, start[f][n], len(outs[n]), max(map(outs[n].count, outs[n]), default=0)) for n, l in enumerate(degrees[f])))
        self.axes = role

    def struct(self, channels: Tuple[int, int, int]) -> "_lib.UvwRoleStruct":
        """``channels``: of the output and the two operands of the layer, whose weights are (paths, C1, C2, C_out)."""
        stride = {1: channels[2] * channels[0], 2: channels[0], 0: 1}
        o, s, f = self.axes
        return _lib.UvwRoleStruct(self.data_ptr, C.addressof(self.groups), len(self.table), len(self.groups), *self.dims, channels[s],
                                  channels[f], channels[o], stride[s], stride[f], stride[o], channels[0] * channels[1] * channels[2])


class UvwPlan:
    """Device tables of one layer.  ``paths``: (k, i, j) of every weight - output, first and second operand irrep - and
    ``scales`` the factors on their Clebsch-Gordan blocks."""

    def __init__(self, paths, scales, irreps_out, irreps1, irreps2, device):
        self.device = torch.device(device)
        degrees = [[ir.l for ir in irs] for irs in (irreps_out, irreps1, irreps2)]
        self.usable = (len(paths) > 0 and all(0 <= l <= TRIPLE_MAX_L for ls in degrees for l in ls)
                       and all(abs(degrees[1][i] - degrees[2][j]) <= degrees[0][k] <= degrees[1][i] + degrees[2][j] for k, i, j in paths))
        if not self.usable:
            return
        start = [np.cumsum([0] + [2 * l + 1 for l in ls]).tolist() for ls in degrees]
        self.dims = tuple(s[-1] for s in start)
        self.num_paths = len(paths)
        self.roles = {role: _Role(role, paths, scales, degrees, start) for role in (FORWARD, GRAD_1, GRAD_2)}
        self.blob = torch.from_numpy(np.concatenate([r.table for r in self.roles.values()]).view(np.uint8)).to(device)
        for n, r in enumerate(self.roles.values()):
            r.data_ptr = self.blob.data_ptr() + n * self.num_paths * _PATH.itemsize
        self._structs, self._fits = {}, {}
        status_flag(self.device)          # now: a call under capture would take it from the graph's memory

    def structs(self, channels: Tuple[int, int, int], roles):
        key = (channels, roles)
        if key not in self._structs:
            self._structs[key] = (_lib.UvwRoleStruct * len(roles))(*(self.roles[r].struct(channels) for r in roles))
        return self._structs[key]

    def supported(self, x1: Tensor, x2: Tensor, w: Tensor) -> bool:
        if not (self.usable and x1.is_cuda and x1.dtype == x2.dtype == w.dtype == torch.float32 and x1.ndim == 3 and x2.ndim == 3
                and x1.shape[0] == x2.shape[0] and x1.shape[0] > 0 and w.ndim == 4
                and w.shape[:3] == (self.num_paths, x1.shape[2], x2.shape[2])
                and (x1.shape[1], x2.shape[1]) == self.dims[1:] and x1.device == x2.device == w.device == self.device):
            return False
        key = (w.shape[1:], x1.shape[0])
        if key not in self._fits:
            channels = (w.shape[3], w.shape[1], w.shape[2])
            if len(self._fits) > 256:
                self._fits.clear()
            lib, (forward,) = _lib.lib(), self.structs(channels, (FORWARD,))
            self._fits[key] = (all(lib.eqt_uvw_scratch_floats(self.structs(channels, (r,)), 1, x1.shape[0]) >= 0 for r in self.roles)
                               and lib.eqt_uvw_wgrad_scratch_floats(C.byref(forward), self.roles[FORWARD].degrees, x1.shape[0]) >= 0)
        return self._fits.get(key, False) and (x1.data_ptr() | x2.data_ptr() | w.data_ptr()) % 16 == 0


def uvw_contract(plan: UvwPlan, operands: Sequence[Optional[Tensor]], w: Tensor, roles, limit: int) -> list:
    """The products of ``roles`` (at most two; both run in one launch where their outputs have equally many channels and one
    launch has room for them), from contiguous ``operands`` = (gradient of the output, first, second operand) and the weights.
    Partial outputs and transposed operands take some 12 to 60 KB a sample; batches whose scratch would exceed ``limit`` bytes run in
    slices of whole sample tiles."""
    n = next(t for t in operands if t is not None).shape[0]
    channels = (w.shape[3], w.shape[1], w.shape[2])
    structs, lib, dev = plan.structs(channels, roles), _lib.lib(), w.device
    with _lib.on_device(dev):
        together = len(roles) == 1 or channels[roles[0][0]] == channels[roles[1][0]]
        floats = int(lib.eqt_uvw_scratch_floats(structs, len(roles), n)) if together else -1
        if floats < 0 and len(roles) == 2:
            return [uvw_contract(plan, operands, w, (r,), limit)[0] for r in roles]
        outs = [w.new_empty(n, plan.dims[r[0]], channels[r[0]]) for r in roles]
        step = n
        if 4 * floats > limit:
            step = min(n, max(_TILE, n // -(-4 * floats // limit) // _TILE * _TILE))
            floats = max(int(lib.eqt_uvw_scratch_floats(structs, len(roles), m)) for m in (step, (n - 1) % step + 1))
        scratch = torch.empty(max(floats, 0), dtype=torch.float32, device=dev)        # of this call: calls on other streams may overlap it
        for a in range(0, n, step):
            pointers = [(C.c_void_p * len(roles))(*(t.data_ptr() + 4 * a * t.shape[1] * t.shape[2] for t in ts)) for ts in (
                [operands[r[1]] for r in roles], [operands[r[2]] for r in roles], outs)]
            _lib.check(lib.eqt_uvw_contract(structs, len(roles), *pointers, w.data_ptr(), scratch.data_ptr(), floats, min(step, n - a),
                                            status_flag(dev).data_ptr(), _lib.stream_ptr(dev)), "eqt_uvw_contract")
    return outs


def uvw_wgrad(plan: UvwPlan, x1: Tensor, x2: Tensor, grad: Tensor) -> Tensor:
    """Gradient of the weights, (paths, C1, C2, C_out), from contiguous operands."""
    channels = (grad.shape[2], x1.shape[2], x2.shape[2])
    role, degrees = plan.structs(channels, (FORWARD,)), plan.roles[FORWARD].degrees
    gw, n, lib, dev = grad.new_empty(plan.num_paths, *channels[1:], channels[0]), grad.shape[0], _lib.lib(), grad.device
    with _lib.on_device(dev):
        floats = int(lib.eqt_uvw_wgrad_scratch_floats(role, degrees, n))
        scratch = torch.empty(max(floats, 0), dtype=torch.float32, device=dev)
        _lib.check(lib.eqt_uvw_wgrad(role, degrees, x1.data_ptr(), x2.data_ptr(), grad.data_ptr(), gw.data_ptr(), scratch.data_ptr(), floats,
                                     n, status_flag(dev).data_ptr(), _lib.stream_ptr(dev)), "eqt_uvw_wgrad")
    return gw
