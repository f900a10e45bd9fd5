"""Tensor-core paths of the indexed products with an operand shared by the batch.

``indexed_vecmat_scale_gather`` with a 3-D matrix operand and ``indexed_outer_scale_gather`` with
``out_accumulated=True`` are GEMMs over the batch; for float32 operands with channel counts that are multiples of 32
they run on tcgen05 (``eqt_vecmat_tc_grouped`` / ``eqt_outer_tc_grouped``) instead of the table-driven CUDA-core kernels.  What the
kernels need besides the operands depends on the index tables only (k-block columns, packing of entries into
128-row slices, reduction lists) and is built once per table and device and cached.
"""
from __future__ import annotations

import ctypes as C
import threading
from collections import OrderedDict
from typing import Optional

import numpy as np
import torch
from torch import Tensor

from .. import _lib
from .mix_tc_op import status_flag

MIN_BATCH = 512          # below this the table-driven kernels are as fast and have no set-up cost
MAX_COLUMNS = 128        # widest output row of a GEMM: its accumulators have to fit tensor memory beside the split operand
MAX_PLANS = 256
_plans: "OrderedDict[tuple, tuple]" = OrderedDict()
_plans_lock = threading.Lock()


def _cached(kind, dev, tensors, extra, build):
    """Plan for these index tensors.  A plan is keyed by the identity and version of the tensors it was built from
    and keeps them alive, so that neither a recycled address nor an in-place update can alias another table; the
    tables of a module are persistent buffers, so layers hit the cache on every call after the first.

    ``None`` where no plan can be had and the table-driven kernels have to run: building one copies the tables to the host,
    which a stream that is being captured does not allow, and tensors of inference mode have no version."""
    if any(t is not None and t.is_inference() for t in tensors):
        return None
    key = (kind, dev, tuple(None if t is None else (id(t), t._version) for t in tensors)) + tuple(extra)
    with _plans_lock:
        hit = _plans.get(key)
        if hit is not None:
            _plans.move_to_end(key)
            return hit[0]
    if torch.cuda.is_current_stream_capturing():
        return None
    plan = build()
    with _plans_lock:
        _plans[key] = (plan, tensors)
        if len(_plans) > MAX_PLANS:
            _plans.popitem(last=False)
    return plan


def _host(t: Optional[Tensor], default: np.ndarray) -> np.ndarray:
    return default if t is None else t.detach().cpu().numpy()


def _same_reads(reads):
    """Classes of rows that read the same rows, ``{(what they read, sorted): [rows]}``, in order of first appearance;
    ``reads[r]`` lists what row r reads, repeats included."""
    classes: "OrderedDict[tuple, list]" = OrderedDict()
    for row, r in enumerate(reads):
        classes.setdefault(tuple(sorted(r)), []).append(row)
    return classes


class VecmatPlan:
    """Output rows that read the same input rows share work items of up to ``group`` rows (see ``eqt_vecmat_tc_grouped``)."""

    def __init__(self, index1, seg, entries: int, num_out: int, cin: int, cout: int, dev):
        chunks = cin // 32
        sg = _host(seg, np.arange(num_out + 1, dtype=np.int64))
        i1 = _host(index1, np.arange(entries if entries >= 0 else sg[-1], dtype=np.int64))
        classes = _same_reads([i1[sg[r]:sg[r + 1]].tolist() for r in range(num_out)])

        # A k-block costs 16 KB of x and 256 bytes of weights per column.  With the one-row groups at 413 entries of 32 x 32
        # (l = 0..6) a pass moved 9.9 MB per 128 samples and issued 4956 small MMAs; four rows a group make it 5.5 MB and 1368.
        def cost(g):
            return sum(-(-len(rows) // g) * len(reads) for reads, rows in classes.items()) * (64 + g * cout)
        sizes = [1] + [g for g in (2, 3, 4) if cout % 32 == 0 and g * cout <= 128]
        self.group = min(sizes, key=cost)
        group_rows, slot_entry, a_col, kb_begin = [], [], [], [0]
        for reads, rows in classes.items():
            for k in range(0, len(rows), self.group):
                part = rows[k:k + self.group]
                group_rows.append(part + [-1] * (self.group - len(part)))
                # the j-th of the sorted reads of every row of the class is the same input row
                order = [sg[r] + np.argsort(i1[sg[r]:sg[r + 1]], kind="stable") for r in part]
                for j, row1 in enumerate(reads):
                    slot_entry.append([int(o[j]) for o in order] + [-1] * (self.group - len(part)))
                    a_col += [row1 * cin + ch * 32 for ch in range(chunks)]
                kb_begin.append(len(a_col))
        self.slots, self.num_groups = len(slot_entry), len(group_rows)
        self.longest = max((len(reads) * chunks for reads in classes), default=0)

        def dev_i32(v):
            return torch.tensor(v if len(v) else [0], dtype=torch.int32, device=dev)
        self.kb_begin, self.a_col = dev_i32(kb_begin), dev_i32(a_col)
        self.group_rows, self.slot_entry = dev_i32(group_rows), dev_i32(slot_entry)


def vecmat_supported(x: Tensor, w: Tensor, gather_index, index_out, out_accumulated, out_size, num_out) -> bool:
    return (x.is_cuda and x.dtype == torch.float32 and w.dtype == torch.float32 and x.ndim == 3 and w.ndim == 3
            and gather_index is None and index_out is None and not out_accumulated and out_size == num_out
            and x.shape[0] >= MIN_BATCH and x.shape[2] % 32 == 0 and w.shape[2] % 16 == 0 and w.shape[2] <= MAX_COLUMNS
            and x.data_ptr() % 16 == 0)


def _entries(index1, index2, seg, num_out: int) -> int:
    return (index1.shape[0] if index1 is not None else index2.shape[0] if index2 is not None
            else num_out if seg is None else -1)          # -1: as many as the last segment ends at, read with the plan


def vecmat_tc(x: Tensor, w: Tensor, scale, index1, index2, seg, num_out: int) -> Optional[Tensor]:
    """``out[i, M, :] = sum_{t in seg[M]} scale[t] x[i, index1[t], :] @ w[index2[t]]`` on tensor cores; ``None`` without a plan."""
    dev = x.device
    n, rows1, cin = x.shape
    cout = w.shape[2]
    entries = _entries(index1, index2, seg, num_out)
    plan = _cached("vecmat", dev, (index1, seg), (entries, num_out, cin, cout),
                   lambda: VecmatPlan(index1, seg, entries, num_out, cin, cout, dev))
    if plan is None:
        return None
    packed = torch.empty(2, max(plan.slots, 1) * cin * plan.group * cout, dtype=torch.float32, device=dev)
    out = torch.empty(n, num_out, cout, dtype=torch.float32, device=dev)
    with _lib.on_device(dev):
        _lib.check(_lib.lib().eqt_vecmat_tc_grouped(x.data_ptr(), w.data_ptr(), _lib.ptr(index2), _lib.ptr(scale),
                                                    packed[0].data_ptr(), packed[1].data_ptr(), out.data_ptr(), n, rows1, cin, cout,
                                                    num_out, plan.slots, plan.group, plan.num_groups, plan.group_rows.data_ptr(),
                                                    plan.slot_entry.data_ptr(), plan.kb_begin.data_ptr(), plan.a_col.data_ptr(),
                                                    plan.longest, status_flag(dev).data_ptr(), _lib.stream_ptr(dev)), "eqt_vecmat_tc_grouped")
    return out


class OuterPlan:
    """Packing of the entries of an accumulated outer product into 128-row slices (see ``eqt_outer_tc_grouped``): second
    operand rows that meet the same rows of the first share slices, ``group`` of them at a time.  ``swapped``: the operands
    change places and the result is written transposed."""

    def __init__(self, scale, index1, index2, seg, entries: int, num_w: int, c1: int, c2: int, dev):
        sg = _host(seg, np.arange(num_w + 1, dtype=np.int64))
        entries = entries if entries >= 0 else int(sg[-1])
        i1 = _host(index1, np.arange(entries, dtype=np.int64))
        i2 = _host(index2, np.arange(entries, dtype=np.int64))
        sc = _host(scale, np.ones(entries, dtype=np.float32)).astype(np.float32)
        w_of = np.repeat(np.arange(num_w), np.diff(sg))

        def classes_of(first, second):
            rows = np.unique(second)
            meets = {int(r): np.nonzero(second == r)[0] for r in rows}
            return rows, meets, _same_reads([sorted(set(first[meets[int(r)]].tolist())) for r in rows])

        # For every sample a slice reads and splits four 128-byte columns of the first operand and c / 32 per row of the second.
        # The four columns of a slice meet all its second-operand rows, so 64 channels against 128 fill it only the other way
        # round (50k nodes, 64 -> 128 channels: 257 us as they come, 149 us swapped).
        def cost(classes, c_first, c_second, g):
            return sum(-(-len(reads) * c_first // 128) * -(-len(rows) // g) for reads, rows in classes.items()) * (4 + g * c_second // 32)
        options = []
        for swapped, (first, second, cf, cs) in enumerate(((i1, i2, c1, c2), (i2, i1, c2, c1))):
            if cs <= 128:
                found = classes_of(first, second)
                options += [(cost(found[2], cf, cs, g), swapped, g, found) for g in (1, 2, 3, 4) if g * cs <= 128]
        _, self.swapped, self.group, (rows2, meets, classes) = min(options, key=lambda v: v[:3])
        if self.swapped:
            i1, i2, c1, c2 = i2, i1, c2, c1
        chunks = c1 // 32
        a_cols, b_cols, units = [], [], []            # units: (weight, chunk, slot, scale)
        for reads, rows in classes.items():
            slots = [(r1, ch) for r1 in reads for ch in range(chunks)]
            for k in range(0, len(rows), self.group):
                part = [int(rows2[r]) for r in rows[k:k + self.group]]
                for s0 in range(0, len(slots), 4):
                    tile = len(a_cols) // 4
                    b_cols += [r2 * c2 for r2 in part] + [part[0] * c2] * (self.group - len(part))
                    for q, (r1, ch) in enumerate(slots[s0:s0 + 4]):
                        a_cols.append(int(r1) * c1 + ch * 32)
                        for which, r2 in enumerate(part):
                            units += [(int(w_of[t]), ch, (which << 24) + tile * 4 + q, float(sc[t]))
                                      for t in meets[r2] if i1[t] == r1]
                    a_cols += [0] * (-len(a_cols) % 4)
        self.m_tiles = len(a_cols) // 4
        units.sort(key=lambda u: (u[0], u[1], u[2]))
        keys = np.array([u[0] * chunks + u[1] for u in units], dtype=np.int64)
        red_ptr = np.searchsorted(keys, np.arange(num_w * chunks + 1)).astype(np.int32)

        def dev_i32(v):
            return torch.tensor(v if len(v) else [0], dtype=torch.int32, device=dev)
        self.a_cols, self.b_cols = dev_i32(a_cols), dev_i32(b_cols)
        self.red_ptr = torch.from_numpy(red_ptr).to(dev)
        self.red_slot = dev_i32([u[2] for u in units])
        self.red_scale = torch.tensor([u[3] for u in units] or [0.0], dtype=torch.float32, device=dev)


def outer_supported(a: Tensor, b: Tensor, gather_index, index_out, out_accumulated, out_size, num_out) -> bool:
    return (a.is_cuda and a.dtype == torch.float32 and b.dtype == torch.float32 and a.ndim == 3 and b.ndim == 3
            and out_accumulated and gather_index is None and index_out is None and out_size == num_out
            and a.shape[0] == b.shape[0] and a.shape[0] >= MIN_BATCH and a.shape[2] % 32 == 0 and b.shape[2] % 32 == 0
            and b.shape[2] <= MAX_COLUMNS and a.data_ptr() % 16 == 0 and b.data_ptr() % 16 == 0)


def outer_tc(a: Tensor, b: Tensor, scale, index1, index2, seg, num_w: int) -> Optional[Tensor]:
    """``out[w] = sum_i sum_{t in seg[w]} scale[t] a[i, index1[t], :, None] b[i, index2[t], None, :]`` on tensor cores; ``None``
    without a plan."""
    dev = a.device
    n, rows1, c1 = a.shape
    rows2, c2 = b.shape[1], b.shape[2]
    entries = _entries(index1, index2, seg, num_w)
    plan = _cached("outer", dev, (scale, index1, index2, seg), (entries, num_w, c1, c2),
                   lambda: OuterPlan(scale, index1, index2, seg, entries, num_w, c1, c2, dev))
    if plan is None:
        return None
    out = torch.empty(num_w, c1, c2, dtype=torch.float32, device=dev)
    if plan.swapped:
        a, b, rows1, c1, rows2, c2 = b, a, rows2, c2, rows1, c1
    with _lib.on_device(dev):
        need = int(_lib.lib().eqt_outer_tc_scratch_floats(n, plan.group * c2, max(plan.m_tiles, 1)))
        scratch = torch.empty(max(need, 1), dtype=torch.float32, device=dev)     # of this call: calls on other streams may overlap it
        _lib.check(_lib.lib().eqt_outer_tc_grouped(a.data_ptr(), b.data_ptr(), out.data_ptr(), scratch.data_ptr(), scratch.numel(),
                                                   n, rows1, c1, rows2, c2, plan.group, plan.a_cols.data_ptr(),
                                                   plan.b_cols.data_ptr(), plan.m_tiles, plan.red_ptr.data_ptr(),
                                                   plan.red_slot.data_ptr(), plan.red_scale.data_ptr(), num_w,
                                                   int(plan.swapped), status_flag(dev).data_ptr(), _lib.stream_ptr(dev)), "eqt_outer_tc_grouped")
    return out
