"""``SO3Linear`` evaluated on the edges of a graph and summed into destination nodes, fused.

    out[d] = sum_{e: dst(e) = d}  SO3Linear(node_x[src(e)], y[e]; W)

The reference offers the per-edge layer only; users gather ``node_x[edge_index[0]]`` before it and
scatter-add after it (``equitorch/nn/linears.py:145-187`` surrounded by the
``edge_index`` convention of ``equitorch/transforms/__init__.py:99-101``).  Here the three steps
are one operation, and because the weights are shared by all edges the sum over edges is moved
*in front of* the channel mixing: the CG contraction is accumulated per destination node
(``S[d, r, :]``, one row per (output component, path)) and the ``C_in x C_out`` matrices are
applied once per node instead of once per edge - the result is the same sum, evaluated in a
different order.  The same holds for every gradient:

    grad_W        = sum_d  S[d]^T g[d]                       (node level)
    G[d]          = g[d] W^T                                 (node level, gradient w.r.t. S)
    grad_y[e]     = <CG, node_x[src(e)], G[dst(e)]>          (edge pass, grouped by destination)
    grad_node_x[s]= (sum_{e: src(e)=s} CG' (g[dst(e)], y[e])) W^T   (edge pass grouped by source, then node level)

No per-edge tensor with a channel axis is ever written to memory.
"""
from __future__ import annotations

import os
from typing import Optional

import torch
from torch import Tensor
from torch.autograd import Function

from ... import _profile
from ...graph import EdgeGraph
from ...ops import batched_sparse_dense_op as _ops, indexed_tc_op
from ...ops.fused_tp_op import (INNER_CHANNELS, TpTable, cg_inner, cg_inner_mix, cg_segment_mix, cg_segment_sum, check_status,
                                mix_scratch)
from ...ops.mix_tc_op import (MixPlan, mix_tc, mix_tc_transposed, wgrad_tc, supported as _tc_supported,
                              supported_transposed as _tc_supported_t, supported_wgrad as _tc_supported_w)
from ...structs import TensorProductInfo


# The fused kernels bound every wait on an asynchronous copy; a wait that runs out raises a per-device status
# word and the kernel returns with partial output.  `fused_tp_op.check_status()` turns the word into an
# exception (it synchronises, so it is not called on the hot path); EQT_CHECK_STATUS=1 makes every forward and
# backward of the fused layer call it.
_CHECK_EVERY_CALL = os.environ.get("EQT_CHECK_STATUS", "0") not in ("", "0")


class MixTables:
    """Device tables of a layer's weight step and of its adjoints: ``out[n, M] = sum_{rows r of M} s[n, r] W[path(r)]``.

    ``min_batch``, ``most_columns``: the tensor-core kernels take batches and output widths from / up to these.  Their
    products of TF32 pairs, summed by an adder that truncates, are further from 64 bits than float32 multiply-adds (448 terms,
    64 channels: 1.5e-6 of the norm against 3.6e-7), so a layer whose other route is float32 there keeps to sums that are no
    further: the indexed products with one row an item (2.0e-7; 300 samples, l_max 3, 64 channels 35 us, float32 88 us; 2000
    samples, 128 -> 256 channels 231 and 735 us) where the shapes allow it, the table-driven kernels elsewhere."""

    def __init__(self, info: TensorProductInfo, device, out_dims=None, min_batch: int = 0, most_columns: int = 256):
        self.mix_fwd, self.mix_bwd1, self.mix_bwd2 = (t.to(device) for t in (info.info_M_fwd, info.info_M_bwd1, info.info_M_bwd2))
        # block structure of the weight step for the tensor-core GEMM (None: CUDA-core kernel)
        self.tc_fwd = MixPlan(info.info_M_fwd, out_dims, device) if out_dims is not None else None
        self.min_batch, self.most_columns = min_batch, most_columns
        w, seg = info.info_M_fwd.index2, info.info_M_fwd.seg_out
        self.rows = w.numel() if w is not None else info.info_M_fwd.out_size if seg is None else int(seg[-1])

    def forward(self, s: Tensor, weight: Tensor, mode: str) -> Tensor:
        assert s.shape[1] == self.rows, f"{s.shape[1]} rows for a table of {self.rows}"
        tc, info, (cin, cout) = self._tensor_cores(s, weight.shape[-1]), self.mix_fwd, weight.shape[-2:]
        if (mode == "uv" and tc is None and self.most_columns <= indexed_tc_op.MAX_COLUMNS and s.dtype == torch.float32
                and cin % 32 == 0 and cout % 16 == 0):
            parts = [indexed_tc_op.vecmat_tc(s, w.contiguous(), info.scale, info.index1, info.index2, info.seg_out, info.out_size)
                     for w in weight.split(self.most_columns, dim=-1)]
            if parts[0] is not None:
                return parts[0] if len(parts) == 1 else torch.cat(parts, dim=-1)
        return _mix(s, weight, info, mode, tc)

    def _tensor_cores(self, batch: Tensor, columns: int) -> Optional[MixPlan]:
        return self.tc_fwd if batch.shape[0] >= self.min_batch and columns <= self.most_columns else None

    def grad_weight(self, s: Tensor, grad: Tensor, num_paths: int, mode: str) -> Tensor:
        tcw, b2 = self._tensor_cores(grad, 0), self.mix_bwd2
        if (mode == "uv" and tcw is not None and tcw.regular and grad.dtype == torch.float32
                and _tc_supported_w(s.shape[-1], grad.shape[-1])):
            return wgrad_tc(s, grad, tcw, num_paths)
        if mode == "uv":   # (P, Cout, Cin) summed over nodes, then transposed to the weight's layout
            gw = _ops.indexed_outer_scale_gather(grad, s, b2.scale, b2.index1, b2.index2, b2.seg_out,
                                                 out_accumulated=True, out_size=b2.out_size)
            return gw.transpose(-1, -2).contiguous()
        return _ops.indexed_mul_scale_gather(grad, s, b2.scale, b2.index1, b2.index2, b2.seg_out,
                                             out_accumulated=True, out_size=b2.out_size)

    def grad_inter(self, grad: Tensor, weight: Tensor, mode: str) -> Tensor:
        """Gradient with respect to the intermediate: ``G[n, r] = grad[n, M(r)] W[path(r)]^T``."""
        tc, b1 = self._tensor_cores(grad, weight.shape[-2]), self.mix_bwd1
        if (mode == "uv" and tc is not None and tc.regular
                and _tc_supported_t(weight.shape[-2], weight.shape[-1])):
            return mix_tc_transposed(grad, weight, tc)
        if mode == "uv":
            return _ops.indexed_vecmat_scale_gather(grad, weight.transpose(-1, -2).contiguous(), b1.scale, b1.index2, b1.index1,
                                                    b1.seg_out, out_size=b1.out_size)
        return _ops.indexed_mul_scale_gather(weight, grad, b1.scale, b1.index1, b1.index2, b1.seg_out,
                                             out_size=b1.out_size)


class GraphTPPlan(MixTables):
    """Device tables of one layer for the fused graph kernels (built once per layer and device)."""

    def __init__(self, tp_info_forward: TensorProductInfo, tp_info_backward1: TensorProductInfo,
                 d_in1: int, d_in2: int, d_out: int, device, out_dims=None, in1_dims=None):
        f, b1 = tp_info_forward, tp_info_backward1
        super().__init__(f, device, out_dims)
        self.fwd_table = TpTable(f.info_Mij_fwd, True, d_in1, d_in2, device, f.info_M_fwd)
        # backward-1 tables: input1 is the channel-less operand, input2 the incoming gradient
        self.bwd1_table = TpTable(b1.info_Mij_fwd, False, d_out, d_in2, device, b1.info_M_fwd)
        self.mix_src = b1.info_M_fwd.to(device)
        self.d_in1, self.d_in2, self.d_out = d_in1, d_in2, d_out
        self.device = torch.device(device)
        self.tc_src = MixPlan(b1.info_M_fwd, in1_dims, device) if in1_dims is not None else None
        self._mixed = {}

    def mixed(self, graph: EdgeGraph, node_x: Tensor, weight: Tensor) -> bool:
        """Whether the kernels that mix the rows channel by channel without writing them take these operands of a 'uu' layer."""
        c = node_x.shape[-1]
        if c not in self._mixed:
            self._mixed[c] = c in INNER_CHANNELS and all(mix_scratch(t, 1, c) >= 0 for t in (self.fwd_table, self.bwd1_table))
        return (self._mixed[c] and node_x.shape == (graph.num_src, self.d_in1, c) and node_x.dtype == weight.dtype == torch.float32
                and weight.shape == (self.fwd_table.mix_size[1], c) and graph.num_edges > 0
                and max(graph.num_edges, graph.num_src, graph.num_dst) < 2 ** 31 - 1 and node_x.data_ptr() % 16 == 0
                # sums of many edges on tensor cores pay for writing the rows: 20k nodes, l_max 3, 64 channels, a pass of 100k edges
                # 1416 -> 755 us, of 400k edges 2039 -> 2144
                and (c != 64 or self.d_in1 != 16 or graph.num_edges < 16 * graph.num_dst))


def _mix(s: Tensor, w: Tensor, info, mode: str, tc: "MixPlan | None" = None) -> Tensor:
    if (mode == "uv" and tc is not None and tc.regular and s.dtype == torch.float32
            and _tc_supported(w.shape[-2], w.shape[-1])):
        return mix_tc(s, w, tc)
    op = _ops.indexed_vecmat_scale_gather if mode == "uv" else _ops.indexed_mul_scale_gather
    return op(s, w, info.scale, info.index1, info.index2, info.seg_out, out_size=info.out_size)


class FusedGraphOps:
    """The passes of the fused layer as separate calls, so that a caller can order them (the sharded layer sends halo
    gradients back while the other gradients are computed).  ``state`` is what ``forward`` returns second."""

    def __init__(self, graph: EdgeGraph, plan: GraphTPPlan, mode: str):
        self.graph, self.plan, self.mode = graph, plan, mode

    def forward(self, node_x: Tensor, y: Tensor, weight: Tensor):
        graph, plan = self.graph, self.plan
        with _profile.timed("cg_segment_sum[fwd]"):
            s = cg_segment_sum(plan.fwd_table, node_x, y, graph.src_by_dst, graph.dst_order, graph.dst_ptr,
                               graph.num_dst)
        with _profile.timed("channel_mix[fwd]"):
            out = plan.forward(s, weight, self.mode)
        return out, (node_x, y, weight, s if weight.requires_grad else None)

    def _wt(self, weight: Tensor) -> Tensor:
        return weight.transpose(-1, -2).contiguous() if self.mode == "uv" else weight

    def grad_weight(self, state, grad: Tensor) -> Tensor:
        _, _, weight, s = state
        with _profile.timed("weight_grad"):
            return self.plan.grad_weight(s, grad, weight.shape[0], self.mode)

    def grad_y(self, state, grad: Tensor) -> Tensor:
        node_x, y, weight, _ = state
        graph, plan = self.graph, self.plan
        # gradient w.r.t. the node-level intermediate: G[d, r] = g[d, M(r)] W[w(r)]^T
        with _profile.timed("channel_mix[grad_inter]"):
            g_inter = plan.grad_inter(grad, weight, self.mode)
        with _profile.timed("cg_inner[grad_y]"):
            return cg_inner(plan.fwd_table, node_x, g_inter, graph.src_by_dst, graph.dst_ptr, graph.dst_sorted,
                            graph.dst_order, y.shape[0])

    def grad_x(self, state, grad: Tensor) -> Tensor:
        _, y, weight, _ = state
        graph, plan = self.graph, self.plan
        with _profile.timed("cg_segment_sum[grad_x]"):
            sx = cg_segment_sum(plan.bwd1_table, grad, y, graph.dst_by_src, graph.src_order, graph.src_ptr,
                                graph.num_src)
        with _profile.timed("channel_mix[grad_x]"):
            return _mix(sx, self._wt(weight), plan.mix_src, self.mode, plan.tc_src)

    def backward(self, state, grad: Tensor, need):
        gw = self.grad_weight(state, grad) if need[2] else None
        gy = self.grad_y(state, grad) if need[1] else None
        return self.grad_x(state, grad) if need[0] else None, gy, gw


class MixedGraphOps:
    """The passes of a 'uu' layer where the kernels mix the rows: none of the intermediates exists, and the gradients with
    respect to the features and the weights are one pass (the weights' gradient pairs its rows with the features)."""

    def __init__(self, graph: EdgeGraph, plan: GraphTPPlan):
        self.graph, self.plan = graph, plan

    def forward(self, node_x: Tensor, y: Tensor, weight: Tensor):
        graph = self.graph
        with _profile.timed("cg_segment_sum[fwd]"):
            out, _ = cg_segment_mix(self.plan.fwd_table, node_x, y, graph.src_by_dst, graph.dst_order, graph.dst_ptr, graph.num_dst, weight)
        return out, (node_x, y, weight, None)

    def backward(self, state, grad: Tensor, need):
        node_x, y, weight, _ = state
        graph, plan = self.graph, self.plan
        gx = gy = gw = None
        if need[1]:
            with _profile.timed("cg_inner[grad_y]"):
                gy = cg_inner_mix(plan.fwd_table, node_x, grad, weight, graph.src_by_dst, graph.dst_ptr, graph.dst_order, y.shape[0])
        if need[0] or need[2]:
            with _profile.timed("cg_segment_sum[grad_x]"):
                gx, gw = cg_segment_mix(plan.bwd1_table, grad, y, graph.dst_by_src, graph.src_order, graph.src_ptr, graph.num_src,
                                        weight, node_x if need[2] else None)
        return gx if need[0] else None, gy, gw


class SO3LinearGraphFunction(Function):
    @staticmethod
    def forward(ctx, node_x: Tensor, y: Tensor, weight: Tensor, graph: EdgeGraph, plan: GraphTPPlan, mode: str):
        ctx.ops = MixedGraphOps(graph, plan) if mode == "uu" and plan.mixed(graph, node_x, weight) else FusedGraphOps(graph, plan, mode)
        out, state = ctx.ops.forward(node_x, y, weight)
        ctx.save_for_backward(*state)
        if _CHECK_EVERY_CALL:
            check_status(node_x.device)
        return out

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, grad: Tensor):
        state, ops = ctx.saved_tensors, ctx.ops
        gx, gy, gw = ops.backward(state, grad.contiguous(), ctx.needs_input_grad)
        if _CHECK_EVERY_CALL:
            check_status(grad.device)
        return gx, gy, gw, None, None, None


def so3_linear_graph(node_x: Tensor, y: Tensor, weight: Tensor, graph: EdgeGraph, plan: GraphTPPlan,
                     feature_mode: str = "uv") -> Tensor:
    """Fused gather -> ``SO3Linear`` -> sum over incoming edges.  ``node_x`` (num_src, D1, Cin) float32,
    ``y`` (E, D2) in the caller's edge order, shared ``weight``; returns (num_dst, Dout, Cout)."""
    if weight.ndim != (3 if feature_mode == "uv" else 2):
        raise ValueError("the fused graph layer needs weights shared by all edges")
    return SO3LinearGraphFunction.apply(node_x, y, weight, graph, plan, feature_mode)
