"""Which 'uvw' ``TensorProduct`` calls take the kernels without an intermediate, and that those which do agree with the composed
products over the forms that both accept: views, tables of the caller's own paths, copied, stored and moved layers, streams."""
import copy
import io

import pytest
import torch

from equitorch_b200 import nn as enn
from equitorch_b200.nn.functional.tensor_products import TensorProductUVW, tensor_product_uvw
from equitorch_b200.ops.fused_tp_op import check_status

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
IR = "0e+1o+2e"


def _layer(ir=IR, c=16, **kw):
    return enn.TensorProduct(ir, ir, ir, c, c, c, internal_weights=False, feature_mode="uvw", **kw).to(DEV)


def _operands(layer, n, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    c = layer.weight_shape[1:]
    return [torch.randn(*s, generator=g, device=DEV) for s in ((n, layer.irreps_in1_dim, c[0]), (n, layer.irreps_in2_dim, c[1]), layer.weight_shape,
                                                               (n, layer.irreps_out_dim, c[2]))]


def _composed(layer, x1, x2, w):
    return tensor_product_uvw(x1, x2, w, layer.tp_info_forward, layer.tp_info_backward1, layer.tp_info_backward2)


def _compare(layer, x1, x2, w, cot, taken):
    leaves = [t.detach().requires_grad_(True) for t in (x1, x2, w)]          # detach() keeps strides and address
    out = layer(*leaves)
    assert (type(out.grad_fn).__name__ == TensorProductUVW.__name__ + "Backward") == taken
    got = [out, *torch.autograd.grad(out, leaves, cot)]
    check_status()
    ref = _composed(layer, *leaves)
    for a, b in zip(got, [ref, *torch.autograd.grad(ref, leaves, cot)]):
        assert a.shape == b.shape and float((a - b).norm() / b.norm()) < 3e-6      # the composed sums of 256 terms and more
    return got


@pytest.mark.parametrize("n", [70, 900])
@pytest.mark.parametrize("form", ["contiguous", "transposed", "every_other", "expanded_gradient", "misaligned"])
def test_views(form, n):
    layer = _layer()
    x1, x2, w, cot = _operands(layer, n)
    if form == "transposed":
        x1, w = x1.transpose(1, 2).contiguous().transpose(1, 2), w.permute(3, 0, 2, 1).contiguous().permute(1, 3, 2, 0)
    elif form == "every_other":
        x2 = x2.repeat_interleave(2, dim=0)[::2]
    elif form == "expanded_gradient":
        cot = cot[:1].expand(n, -1, -1)
    elif form == "misaligned":
        x2 = torch.cat([x2.flatten().new_zeros(1), x2.flatten()])[1:].view_as(x2)
        assert x2.data_ptr() % 16
    _compare(layer, x1, x2, w, cot, taken=form != "misaligned")


@pytest.mark.parametrize("kw", [dict(path=[(2, 1, 1), (0, 0, 0), (2, 1, 1), (1, 0, 1), (0, 2, 2)]), dict(path=[(1, 1, 2)], path_norm=False),
                                dict(channel_norm=True)])
def test_paths_and_norms(kw):
    layer = _layer(**kw)
    _compare(layer, *_operands(layer, 333), taken=True)


@pytest.mark.parametrize("ir1,ir2,ir_out,c,taken", [
    ("0e", "16x0e", "0e", 16, True), ("0e", "17x0e", "0e", 16, False),              # irreps of the contracted operand
    ("0e+2e", "0e+2e", "12x2e+0e", 16, True), ("0e+2e", "0e+2e", "13x2e", 16, False),     # 61 and 65 output components
    ("2x0e+2x1o+2x2e", "2x0e+2x1o+2x2e", "2x0e+2x1o+2x2e", 32, False),              # 88 paths x 8 channel groups
    ("4x2e", "4x2e", "2e", 16, True), ("5x2e", "5x2e", "2e", 16, False),            # 160 and 200 terms an output element
    ("0e+1o+2e+3o", "0e", "0e", 16, False), (IR, IR, IR, 48, False)])
def test_limits(ir1, ir2, ir_out, c, taken):
    layer = enn.TensorProduct(ir1, ir2, ir_out, c, c, c, internal_weights=False, feature_mode="uvw").to(DEV)
    _compare(layer, *_operands(layer, 150), taken=taken)


def test_copies_keep_the_route_and_edited_tables_leave_it():
    layer = _layer()
    ops = _operands(layer, 200)
    want = _compare(layer, *ops, taken=True)
    stored = io.BytesIO()
    torch.save(layer, stored)
    stored.seek(0)
    for other in (copy.deepcopy(layer), torch.load(stored, weights_only=False), _layer().to("cpu").to(DEV)):
        for a, b in zip(_compare(other, *ops, taken=True), want):
            assert torch.equal(a, b)
    layer.tp_info_forward.info_Mij_fwd.scale.mul_(2.0)
    out = layer(ops[0].requires_grad_(True), *ops[1:3])
    assert type(out.grad_fn).__name__ != TensorProductUVW.__name__ + "Backward"
    assert float((out - 2 * want[0]).norm() / want[0].norm()) < 6e-6


def test_first_call_under_capture_and_two_streams():
    layer = _layer()
    ops = [_operands(layer, 1000, seed) for seed in (1, 2)]
    _layer()(*ops[0][:3])                                               # libraries and flags
    graph, fresh = torch.cuda.CUDAGraph(), _layer()
    torch.cuda.synchronize()
    with torch.no_grad():
        with torch.cuda.graph(graph):
            captured = fresh(*ops[0][:3])
        graph.replay()
        want = [layer(*o[:3]) for o in ops]
        torch.cuda.synchronize()
        assert float((captured - want[0]).norm() / want[0].norm()) < 3e-6
        graph2 = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph2):                                  # the plan is there now: the kernels themselves are captured
            captured = layer(*ops[1][:3])
        captured.zero_()
        graph2.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, want[1])
        streams, got = [torch.cuda.Stream() for _ in ops], [[], []]
        for _ in range(20):
            for k, stream in enumerate(streams):
                with torch.cuda.stream(stream):
                    got[k].append(layer(*ops[k][:3]))
        torch.cuda.synchronize()
    for k in range(2):
        assert all(torch.equal(t, want[k]) for t in got[k])


@pytest.mark.parametrize("n", [40, 600])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_what_is_not_finite_stays_so(value, n):
    """In the samples that it belongs to, and in them alone (an infinity may come out as NaN: a TF32 pair of it holds inf - inf)."""
    layer = _layer(c=32)
    x1, x2, w, cot = _operands(layer, n)
    x1[3, 0, 5], x2[n - 1, 0, 7] = value, value
    leaves = [t.requires_grad_(True) for t in (x1, x2, w)]
    out = layer(*leaves)
    g1, g2, gw = torch.autograd.grad(out, leaves, cot)
    for t, rows in ((out, {3, n - 1}), (g1, {n - 1}), (g2, {3})):
        bad = set(torch.nonzero(~torch.isfinite(t).flatten(1).all(1)).flatten().tolist())
        assert bad == rows
    assert not torch.isfinite(gw).all()


def test_a_plan_brings_its_flag(monkeypatch):
    """The status flag outlives a captured graph, so it must not be made by a call inside one: the plan has it made."""
    from equitorch_b200.ops import fused_tp_op
    monkeypatch.setattr(fused_tp_op, "_status", {})
    layer = _layer(c=16)
    assert layer._path_plan(torch.device(DEV)).usable and torch.device(DEV) in fused_tp_op._status

