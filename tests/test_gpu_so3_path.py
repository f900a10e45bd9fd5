"""``SO3Linear`` through the kernels on straight-line Clebsch-Gordan blocks ('uu': one pass per direction) against the dense float64 oracle: channel counts that give 1 to 64
threads per sample (powers of two and not), batches from one sample (output irreps spread over the grid, smaller
blocks) to several waves, degrees 0 to 3 with even and odd degree sums, shared and per-sample weights, float32 and bfloat16; and a differentiated
backward pass against the composed products."""
import copy
import pickle

import pytest
import torch

from equitorch_b200 import _lib
from equitorch_b200 import nn as enn
from equitorch_b200.nn.functional.linears import tensor_product_u1u, tensor_product_u1v
from equitorch_b200.ops.so3_path_op import PathPlan
from oracle import tensor_products as otp

DEV = "cuda:0"
# float32: an element is a sum of up to 40 terms of random sign, a weight gradient of 40 n; bfloat16: one rounding of the result
BOUND = {torch.float32: 1e-5, torch.bfloat16: 2.0 ** -7}


def _rel(a, b):
    return float((a.detach().double().cpu() - b.detach().double()).abs().max() / b.detach().double().abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("per_sample", [False, True])
@pytest.mark.parametrize("ir,ir_y,n,c", [("0e+1o", "0e+1o", 1, 4), ("0e+1o+2e", "0e+1o+2e", 7, 12), ("0e+1o+2e+3o", "0e+1o+2e+3o", 129, 64),
                                         ("4x0e+2x1o+2e", "0e+1o+2e", 3001, 32), ("0e+1o+2e", "0e+1o+2e", 5003, 48),
                                         ("0e+1o", "0e+1o", 300, 512), ("0o+1e+2e+3e", "0e+1e+2o+3e", 1000, 20), ("0e+1o+2e", "0e+1o+2e", 20001, 16)])
def test_one_pass_kernels(ir, ir_y, n, c, per_sample, dtype):
    g = torch.Generator().manual_seed(n + c)
    layer = enn.SO3Linear(ir, ir_y, ir, c, c, internal_weights=False, feature_mode="uu").to(DEV)
    dim, dim_y, p = layer.irreps_in1_dim, layer.irreps_in2_dim, layer.num_paths
    x, y = torch.randn(n, dim, c, generator=g).to(dtype), torch.randn(n, dim_y, generator=g).to(dtype)
    w = torch.randn(*((n,) if per_sample else ()), p, c, generator=g).to(dtype)
    cot = torch.randn(n, dim, c, generator=g).to(dtype)
    xo, yo, wo = (t.double().requires_grad_(True) for t in (x, y, w))
    want = otp.so3_linear_dense(xo, yo, wo, ir, ir_y, ir, feature_mode="uu")
    want = [want, *torch.autograd.grad(want, [xo, yo, wo], cot.double())]
    xg, yg, wg = (t.to(DEV).requires_grad_(True) for t in (x, y, w))
    before = _lib.launch_count()
    got = layer(xg, yg, wg)
    got = [got, *torch.autograd.grad(got, [xg, yg, wg], cot.to(DEV))]
    assert _lib.launch_count() - before == (2 if per_sample and n > 1 else 3)       # one sample's weights are shared ones
    for a, b in zip(got, want):
        assert a.dtype == dtype and a.shape == b.shape and _rel(a, b) < BOUND[dtype]
    # a gradient for one operand alone, from a copy of the layer
    (gy,) = torch.autograd.grad(copy.deepcopy(layer)(xg.detach(), yg, wg.detach()), [yg], cot.to(DEV))
    assert torch.equal(gy, got[2])


@pytest.mark.gpu
@pytest.mark.parametrize("ir,ir_y,n,c,c_out", [("0e+1o", "0e+1o", 1, 4, 8), ("0e+1o+2e", "0e+1o+2e", 7, 12, 20),
                                               ("0e+1o+2e+3o", "0e+1o+2e+3o", 513, 64, 32), ("4x0e+2x1o+2e", "0e+1o+2e", 1501, 32, 64),
                                               ("0o+1e+2e+3e", "0e+1e+2o+3e", 300, 16, 16), ("0e+1o+2e+3o", "0e+1o+2e+3o", 2003, 128, 48)])
def test_channel_mixing_layer(ir, ir_y, n, c, c_out):
    """'uv' through the row kernels: every degree triple, channel counts with and without a tensor-core GEMM."""
    g = torch.Generator().manual_seed(n + c)
    layer = enn.SO3Linear(ir, ir_y, ir, c, c_out, internal_weights=False, feature_mode="uv").to(DEV)
    dim, dim_y, p = layer.irreps_in1_dim, layer.irreps_in2_dim, layer.num_paths
    x, y, cot = torch.randn(n, dim, c, generator=g), torch.randn(n, dim_y, generator=g), torch.randn(n, dim, c_out, generator=g)
    w = torch.randn(p, c, c_out, generator=g) / c ** 0.5
    xo, yo, wo = (t.double().requires_grad_(True) for t in (x, y, w))
    want = otp.so3_linear_dense(xo, yo, wo, ir, ir_y, ir, feature_mode="uv")
    want = [want, *torch.autograd.grad(want, [xo, yo, wo], cot.double())]
    xg, yg, wg = (t.to(DEV).requires_grad_(True) for t in (x, y, w))
    assert layer._path_plan(xg.device).uv_supported(xg, yg, wg)
    got = layer(xg, yg, wg)
    got = [got, *torch.autograd.grad(got, [xg, yg, wg], cot.to(DEV))]
    for a, b in zip(got, want):
        assert a.shape == b.shape and _rel(a, b) < BOUND[torch.float32]
    (gy,) = torch.autograd.grad(layer(xg.detach(), yg, wg.detach()), [yg], cot.to(DEV))
    assert torch.equal(gy, got[2])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["uu", "uv"])
def test_differentiated_backward_pass(mode):
    g = torch.Generator().manual_seed(0)
    ir, n, c = "0e+1o+2e", 33, 8
    layer = enn.SO3Linear(ir, ir, ir, c, c, internal_weights=False, feature_mode=mode).to(DEV)
    weight = torch.randn(*layer.weight_shape, generator=g)
    leaves = [t.to(DEV).requires_grad_(True) for t in (torch.randn(n, 9, c, generator=g), torch.randn(n, 9, generator=g),
                                                       weight, torch.randn(n, 9, c, generator=g))]
    product = tensor_product_u1u if mode == "uu" else tensor_product_u1v
    infos = (layer.tp_info_forward, layer.tp_info_backward1, layer.tp_info_backward2)

    def second(fn):
        x, y, w, cot = leaves
        first = torch.autograd.grad(fn(x, y, w), [x, y, w], cot, create_graph=True)
        return torch.autograd.grad(sum((t * t).sum() for t in first), leaves)
    for a, b in zip(second(layer), second(lambda x, y, w: product(x, y, w, *infos))):
        assert _rel(a, b.cpu()) < 1e-5


# (irreps, paths, whether the one-pass kernels take them, whether their rows are the rows of the layer's weight step)
PATH_LISTS = [("0e+1e", None, True, True), ("0e+1o+2e+3o", None, True, True), ("0e", None, True, True),
              ("0e+1e", [(1, 0, 1), (1, 1, 0), (0, 0, 0)], True, True), ("2x0e", [(1, 1, 1), (0, 0, 0)], True, True),
              ("0e+1e+2e", [(2, 1, 1), (0, 2, 2), (2, 2, 0), (1, 1, 1), (2, 0, 2)], True, True),
              ("0e+1e", [(1, 1, 0), (0, 0, 0), (1, 1, 0)], True, True),                    # twice, one entry a component
              ("0e+1e", [(1, 1, 1), (1, 1, 1)], True, False), ("0e+1e", [(0, 0, 0), (1, 1, 1), (1, 0, 1), (1, 1, 1)], True, False),
              ("0e+1e", [(0, 0, 0), (1, 0, 0), (0, 1, 1)], False, False)]                  # 0 x 0 -> 1 does not couple


@pytest.mark.parametrize("ir,path,usable,match", PATH_LISTS)
def test_rows_of_the_plan_and_of_the_weight_step(ir, path, usable, match):
    layer = enn.SO3Linear(ir, ir, ir, 8, 8, feature_mode="uv", path=path)
    plan, table = PathPlan(*layer._paths, layer.irreps_out, layer.irreps_in1, layer.irreps_in2, "cpu"), layer.tp_info_forward.info_M_fwd
    assert plan.usable == usable and plan.rows_match(table) == match
    if match:                     # the rows in number and, row by row, in what they are multiplied with
        rows = [w for weights in plan.row_weights for w in weights]
        assert len(rows) == plan.num_rows and rows == (list(range(len(rows))) if table.index2 is None else table.index2.tolist())


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["uu", "uv"])
@pytest.mark.parametrize("n,c", [(5, 8), (600, 32)])
@pytest.mark.parametrize("ir,path,usable,match", PATH_LISTS[:-1])        # the composition refuses the last
def test_path_lists(ir, path, usable, match, n, c, mode):
    g = torch.Generator().manual_seed(n)
    layer = enn.SO3Linear(ir, ir, ir, c, c, internal_weights=False, feature_mode=mode, path=path).to(DEV)
    dim = layer.irreps_in1_dim
    leaves = [torch.randn(n, dim, c, generator=g), torch.randn(n, dim, generator=g), torch.randn(*layer.weight_shape, generator=g)]
    cot = torch.randn(n, dim, c, generator=g)
    lo = [t.double().requires_grad_(True) for t in leaves]
    want = otp.so3_linear_dense(*lo, ir, ir, ir, feature_mode=mode, path=path)
    want = [want, *torch.autograd.grad(want, lo, cot.double())]
    lg = [t.to(DEV).requires_grad_(True) for t in leaves]
    got = layer(*lg)
    got = [got, *torch.autograd.grad(got, lg, cot.to(DEV))]
    for a, b in zip(got, want):
        assert a.shape == b.shape and _rel(a, b) < BOUND[torch.float32]


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["uu", "uv"])
@pytest.mark.parametrize("n,c,per_sample", [(33, 8, False), (600, 32, False), (33, 8, True)])
def test_second_derivatives_with_operands_that_are_views(mode, n, c, per_sample):
    """A transposed x, a slice as y and a strided weight: gradients of the energy and of a loss on them (training on forces)
    against the composed products."""
    g = torch.Generator().manual_seed(n)
    ir = "0e+1o+2e"
    layer = enn.SO3Linear(ir, ir, ir, c, c, internal_weights=False, feature_mode=mode).to(DEV)
    shape = ((n,) if per_sample else ()) + tuple(layer.weight_shape)
    leaves = [t.to(DEV).requires_grad_(True) for t in (torch.randn(n, c, 9, generator=g), torch.randn(n, 13, generator=g),
                                                       torch.randn(*shape, generator=g), torch.randn(n, 9, c, generator=g))]
    product = tensor_product_u1u if mode == "uu" else tensor_product_u1v
    infos = (layer.tp_info_forward, layer.tp_info_backward1, layer.tp_info_backward2)

    def both(fn):
        x0, y0, w0, cot = leaves
        x, y, w = x0.transpose(1, 2), y0[:, 4:], torch.cat([w0, w0], dim=-1)[..., :c]
        assert not (x.is_contiguous() or y.is_contiguous() or w.is_contiguous())
        first = torch.autograd.grad(fn(x, y, w), [x0, y0, w0], cot, create_graph=True)
        return [t.detach() for t in first] + list(torch.autograd.grad(sum((t * t).sum() for t in first), leaves))
    for a, b in zip(both(layer), both(lambda x, y, w: product(x, y, w, *infos))):
        assert _rel(a, b.cpu()) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("mode,dtype,per_sample", [("uu", torch.float32, False), ("uu", torch.bfloat16, True), ("uv", torch.float32, False)])
def test_gradients_of_some_operands(mode, dtype, per_sample):
    """Every subset of operands that want a gradient: the same values, and no operand is kept that none of them takes."""
    g = torch.Generator().manual_seed(5)
    ir, n, c = "0e+1o+2e", 601, 32
    layer = enn.SO3Linear(ir, ir, ir, c, c, internal_weights=False, feature_mode=mode).to(DEV)
    shape = ((n,) if per_sample else ()) + tuple(layer.weight_shape)
    values = [torch.randn(*s, generator=g).to(dtype).to(DEV) for s in ((n, 9, c), (n, 9), shape)]
    cot = torch.randn(n, 9, c, generator=g).to(dtype).to(DEV)

    def run(wanted, after=lambda out, operands: None):
        operands = [v.clone().requires_grad_(k in wanted) for k, v in enumerate(values)]
        out = layer(*operands)
        after(out, operands)
        return dict(zip(wanted, torch.autograd.grad(out, [operands[k] for k in wanted], cot)))
    full = run((0, 1, 2))
    for wanted in ((0,), (1,), (2,), (0, 1), (0, 2), (1, 2)):
        part = run(wanted)
        assert all(torch.equal(part[k], full[k]) for k in wanted)
    if mode == "uv":                   # the rows are kept for the weight gradient, so that x may change in place
        assert torch.equal(run((2,), lambda out, operands: operands[0].mul_(2))[2], full[2])


def _norm_errors(mode, ir, n, c, c_out, per_sample=False):
    """2-norm errors of output and gradients against the layer in float64, over the norms."""
    g = torch.Generator().manual_seed(n + c + c_out)
    layer = enn.SO3Linear(ir, ir, ir, c, c_out, internal_weights=False, feature_mode=mode).to(DEV)
    dim, shape = layer.irreps_in1_dim, ((n,) if per_sample else ()) + tuple(layer.weight_shape)
    leaves = [torch.randn(n, dim, c, generator=g), torch.randn(n, dim, generator=g), torch.randn(*shape, generator=g) * (c ** -0.5 if mode == "uv" else 1)]
    cot = torch.randn(n, dim, c_out, generator=g)
    results = []
    for dtype, call in ((torch.float32, layer), (torch.float64, lambda x, y, w: otp.so3_linear_dense(x, y, w, ir, ir, ir, feature_mode=mode))):
        lv = [t.to(dtype).to(DEV).requires_grad_(True) for t in leaves]
        out = call(*lv)
        results.append([out.detach(), *torch.autograd.grad(out, lv, cot.to(dtype).to(DEV))])
    return [float((a.double() - b).norm() / b.norm()) for a, b in zip(*results)]


@pytest.mark.gpu
@pytest.mark.parametrize("ir,n,c,c_out,bounds", [("0e+1o+2e+3o", 300, 64, 64, (5e-7, 4.5e-7, 2.5e-7, 3.5e-7)),
                                                 ("0e+1o+2e+3o", 511, 128, 128, (7e-7, 6.5e-7, 3.5e-7, 5e-7)),
                                                 ("0e+1o+2e+3o", 2000, 64, 256, (5e-7, None, None, None)),
                                                 ("0e+1o+2e+3o", 2000, 256, 64, (None, 4.5e-7, 2.7e-7, None))])
def test_channel_mixing_in_float32_where_it_was(ir, n, c, c_out, bounds):
    """Batches below the tensor-core kernels' and outputs wider than theirs: sums of float32 multiply-adds.  The bounds are 1.3
    to 1.4 times the errors of the composed products (3.6e-7, 3.4e-7, 1.8e-7, 2.4e-7 at 300 samples); the tensor cores'
    are 1.5 to 5 times those."""
    for e, bound in zip(_norm_errors("uv", ir, n, c, c_out), bounds):
        assert bound is None or e < bound


@pytest.mark.gpu
@pytest.mark.parametrize("ir,n,c,c_out,bound", [("0e+1o+2e+3o", 700, 128, 128, 4e-6), ("0e+1o+2e+3o", 700, 128, 64, 4e-6),
                                                ("8x0e+4x1o+4x2e", 600, 32, 32, 4e-6), ("8x0e+4x1o+4x2e", 520, 64, 96, 4e-6)])
def test_long_sums_are_added_up_in_pieces(ir, n, c, c_out, bound):
    """Sums of 16 to 112 k-blocks of 32 terms: no further from 64 bits than pieces of 16 in one accumulator.  Bound: 192
    truncated additions of 1.7e-8 of the norm each and the split's 6.5e-8, 3.3e-6, and a fifth for the draw (the composed
    products are at 3.2e-6 with 28 k-blocks; in one piece 5.6e-6, growing with the length)."""
    assert _norm_errors("uv", ir, n, c, c_out)[0] < bound


@pytest.mark.gpu
@pytest.mark.parametrize("ir,n,c,per_sample,composed", [("0e+1o+2e+3o", 1001, 64, False, (7.5e-8, 7.6e-8, 9.9e-8, 1.5e-7)),
                                                        ("0e+1o+2e", 4001, 32, True, (6.4e-8, 6.4e-8, 8.8e-8, 6.1e-8))])
def test_channelwise_sums_are_no_further_from_64_bits(ir, n, c, per_sample, composed):
    """Against the errors of the composed products on such operands; a tenth for other draws of them."""
    for e, bound in zip(_norm_errors("uu", ir, n, c, c, per_sample), composed):
        assert e < 1.1 * bound


def _composed(layer, x, y, w):
    product = tensor_product_u1u if layer.feature_mode == "uu" else tensor_product_u1v
    return product(x, y, w, *layer._tables())


def _small_layer(mode, n=100, c=32, seed=0):
    g = torch.Generator().manual_seed(seed)
    ir = "0e+1o+2e"
    layer = enn.SO3Linear(ir, ir, ir, c, c, internal_weights=False, feature_mode=mode).to(DEV)
    return layer, [t.to(DEV) for t in (torch.randn(n, 9, c, generator=g), torch.randn(n, 9, generator=g),
                                       torch.randn(*layer.weight_shape, generator=g))]


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["uu", "uv"])
def test_first_call_while_a_stream_is_captured(mode):
    """A layer whose tables are not on the device yet takes the composed products, as before there were one-pass kernels."""
    warm, operands = _small_layer(mode, seed=1)
    want = _composed(warm, *operands).clone()
    layer, _ = _small_layer(mode)
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad():
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            got = layer(*operands)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    assert layer._path_plans == {} and _rel(layer(*operands), want.cpu()) < 1e-5 and layer._path_plans != {}


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["uu", "uv"])
def test_tables_that_are_exchanged_written_to_or_stored(mode):
    layer, operands = _small_layer(mode)
    want = layer(*operands).cpu()
    for other in (copy.deepcopy(layer), pickle.loads(pickle.dumps(layer)), copy.deepcopy(layer).cpu().to(DEV)):
        assert other._is_own() and torch.equal(other(*operands).cpu(), want)
    stored = layer.__getstate__()                      # as a layer is stored that knows nothing of the one-pass kernels
    for name in ("_paths", "_own"):
        del stored[name]
    old = enn.SO3Linear.__new__(enn.SO3Linear)
    old.__setstate__(stored)
    assert _rel(old(*operands), want) < 1e-5 and old._path_plans == {}
    old = old.to("cpu").to(DEV)
    assert _rel(old(*operands), want) < 1e-5
    layer.tp_info_forward.info_Mij_fwd.scale.mul_(2)   # written to in place
    assert not layer._is_own() and _rel(layer(*operands), 2 * want) < 1e-5
    layer, _ = _small_layer(mode)
    scale = layer.tp_info_forward.info_Mij_fwd.scale
    layer.tp_info_forward = layer.tp_info_forward._replace(info_Mij_fwd=layer.tp_info_forward.info_Mij_fwd._replace(scale=3 * scale))
    assert _rel(layer(*operands), 3 * want) < 1e-5
