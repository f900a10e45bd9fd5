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
                and max(graph.num_edges, graph.num_src, graph.num_dst) < 2 ** 31 - 1 and node_x.data_ptr() % 16 == 0)


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


class ChannelwiseGraphOps(FusedGraphOps):
    """The passes of a 'uu' layer where the kernels can mix the rows: a pass writes rows only where that is faster.

    Mixing saves writing and reading the rows, which counts with few edges a node; where the edges count, a pass without rows is
    the slower one at l_max 3 (sums of 64 channels run on tensor cores, others on four warps a node), and the weights' gradient
    costs a walk over all edges, shared with the features' gradient, unless the rows of the forward pass are kept.  The limits are
    the crossings of both forms over 100 to 100k nodes of 2 to 60 edges.  l_max 3, us, with rows / mixed: forward pass of 30k nodes, 64
    channels, of 8 edges 649 / 551, of 12 672 / 760; forward pass and the gradients of features and weights, 10k nodes, 128 channels, of 20 edges
    1555 / 1460, of 30 2058 / 2099, of 60 3560 / 3965; forward pass and the weights' gradient alone, l_max 2, 32 channels, 10k nodes of 8
    edges 56 / 57, of 15 70 / 85."""

    def __init__(self, graph: EdgeGraph, plan: GraphTPPlan, channels: int, need_x: bool, need_weight: bool):
        super().__init__(graph, plan, "uu")
        nodes, edges, high = graph.num_dst, graph.num_edges, plan.d_in1 == 16
        out, x, kept = self._rows_from(channels, nodes)
        self.keeps = need_weight and (high and edges >= kept * nodes if need_x else self._kept_alone(channels))
        self.out_rows = self.keeps or (high and edges >= out * nodes)
        self.x_rows = high and edges >= x * graph.num_src
        # four warps share the adjoint of a node in a small graph (300 nodes, 4 edges: l_max 2, 32 channels 8.6 / 9.1)
        self.y_rows = nodes <= 400 and channels == (128 if plan.d_in1 == 4 else 32)

    @staticmethod
    def _rows_from(channels: int, nodes: int):
        """Edges a node from which rows are written at l_max 3: in the forward pass, in the gradient of the features alone, and in
        a forward pass that keeps them for the weights' gradient beside the features'."""
        if channels == 16:       # few nodes leave SMs idle, and then edges cost little
            return (60, 60, 60) if nodes < 450 else (25, 25, 45) if nodes < 1500 else (9, 10, 24)
        # 128: from 100 nodes an SM on the sums' rows come from four warps a node, which gain less over a walk that mixes them
        return {32: (16, 10, 18), 64: (11, 11, 13), 128: (16, 9, 24 if nodes < 14_800 else 45)}[channels]

    def _kept_alone(self, channels: int) -> bool:
        """Whether keeping the rows is faster than a walk for the weights' gradient alone: a matter of their bytes (L2 holds 126 MB)."""
        nodes, edges = self.graph.num_dst, self.graph.num_edges
        size = nodes * channels * self.plan.fwd_table.num_rows * 4
        if self.plan.d_in1 == 16:
            return size < 64e6 or edges >= (5 if channels in (32, 64) else 4) * nodes
        return edges >= (3 if nodes >= 900 and size < 16e6 else 8 if 1e6 <= size < 48e6 else 13) * nodes

    def forward(self, node_x: Tensor, y: Tensor, weight: Tensor):
        if self.out_rows:
            out, state = super().forward(node_x, y, weight)
            return out, state if self.keeps else (*state[:3], None)
        graph = self.graph
        with _profile.timed("cg_segment_sum[fwd]"):
            out, _ = cg_segment_mix(self.plan.fwd_table, node_x, y, graph.src_by_dst, graph.dst_order, graph.dst_ptr, graph.num_dst, weight)
        return out, (node_x, y, weight, None)

    def grad_y(self, state, grad: Tensor) -> Tensor:
        if self.y_rows:
            return super().grad_y(state, grad)
        node_x, y, weight, _ = state
        graph = self.graph
        with _profile.timed("cg_inner[grad_y]"):
            return cg_inner_mix(self.plan.fwd_table, node_x, grad, weight, graph.src_by_dst, graph.dst_ptr, graph.dst_order, y.shape[0])

    def grad_x(self, state, grad: Tensor) -> Tensor:
        return super().grad_x(state, grad) if self.x_rows else self._walk_sources(state, grad, False)[0]

    def _walk_sources(self, state, grad: Tensor, with_weight: bool):
        node_x, y, weight, _ = state
        graph = self.graph
        with _profile.timed("cg_segment_sum[grad_x]"):
            return cg_segment_mix(self.plan.bwd1_table, grad, y, graph.dst_by_src, graph.src_order, graph.src_ptr, graph.num_src,
                                  weight, node_x if with_weight else None)

    def backward(self, state, grad: Tensor, need):
        if not need[2] or self.keeps:
            return super().backward(state, grad, need)
        gy = self.grad_y(state, grad) if need[1] else None
        gx, gw = self._walk_sources(state, grad, True)
        return gx if need[0] else None, gy, gw


class SO3LinearGraphFunction(Function):
    @staticmethod
    def forward(ctx, node_x: Tensor, y: Tensor, weight: Tensor, graph: EdgeGraph, plan: GraphTPPlan, mode: str, with_grad: bool):
        if mode == "uu" and plan.mixed(graph, node_x, weight):
            ctx.ops = ChannelwiseGraphOps(graph, plan, node_x.shape[-1], with_grad and node_x.requires_grad, with_grad and weight.requires_grad)
        else:
            ctx.ops = FusedGraphOps(graph, plan, mode)
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
        return gx, gy, gw, None, None, None, None


def so3_linear_graph(node_x: Tensor, y: Tensor, weight: Tensor, graph: EdgeGraph, plan: GraphTPPlan,
                     feature_mode: str = "uv") -> Tensor:
    """Fused gather -> ``SO3Linear`` -> sum over incoming edges.  ``node_x`` (num_src, D1, Cin) float32,
    ``y`` (E, D2) in the caller's edge order, shared ``weight``; returns (num_dst, Dout, Cout)."""
    if weight.ndim != (3 if feature_mode == "uv" else 2):
        raise ValueError("the fused graph layer needs weights shared by all edges")
    return SO3LinearGraphFunction.apply(node_x, y, weight, graph, plan, feature_mode, torch.is_grad_enabled())
