"""'uvw' ``TensorProduct`` without an intermediate (tensor-core contraction of one operand with the weights, the other operand and the
Clebsch-Gordan blocks in the epilogue; weight gradient on float32 multiply-adds or on tensor cores) against the dense float64
oracle: sample tiles and chunks of 16 and 32 with remainders, one sample, batches of several waves, 16 and 32 channels on every side, degrees of either parity, repeated irreps, output components that
no path reaches; and the exchange of roles against the blocks themselves."""
import numpy as np
import pytest
import torch

from equitorch_b200 import nn as enn
from equitorch_b200.constants import so3_clebsch_gordan
from equitorch_b200.nn.functional import tensor_products as ftp
from equitorch_b200.nn.functional.tensor_products import TensorProductUVW, tensor_product_uvw
from equitorch_b200.ops.uvw_op import FORWARD, GRAD_1, GRAD_2, exchanged_scale
from oracle import tensor_products as otp

DEV = "cuda:0"


def _rel(a, b):
    return float((a.detach().double().cpu() - b.detach().double()).norm() / b.detach().double().norm())


@pytest.mark.parametrize("degrees", [(0, 0, 0), (1, 1, 0), (0, 2, 2), (2, 1, 1), (1, 1, 1), (2, 2, 1), (2, 2, 2)])
def test_exchanged_roles_are_multiples(degrees):
    ours = so3_clebsch_gordan(*degrees)
    for role in (FORWARD, GRAD_1, GRAD_2):
        block = so3_clebsch_gordan(*(degrees[a] for a in role))
        assert np.abs(ours.transpose(role) - exchanged_scale(degrees, role) * block).max() < 1e-14


@pytest.mark.gpu
@pytest.mark.parametrize("ir1,ir2,ir_out,n,c1,c2,c_out", [
    ("0e+1o", "0e+1o", "0e+1o", 1, 16, 16, 16), ("0e+1o+2e", "0e+1o+2e", "0e+1o+2e", 31, 32, 32, 32),
    ("0e+1o+2e", "0e+1o+2e", "0e+1o+2e", 129, 16, 32, 32), ("0e+1o+2e", "0e+1o+2e", "0e+1o+2e", 2003, 32, 16, 16),
    ("2x0e+1o+1e", "0e+1o+2e+2o", "1e+2x2o+0o+1o", 257, 32, 32, 16), ("0e+1o+2e", "0e+1o+2e", "0e+1o+2e", 20011, 16, 16, 32),
    ("0e", "1o", "1o+2e", 100, 16, 16, 16), ("0e+1o+2e", "0e+1o+2e", "0e+1o+2e", 511, 32, 32, 32), ("0e+1o", "0e+1o", "0e+1o", 512, 32, 32, 32),
    ("0e+1o+2e", "0e+1o+2e", "0e+1o+2e", 300, 16, 32, 32), ("0e+1o+2e", "0e+1o+2e", "0e+1o+2e", 17, 32, 16, 32), ("0e", "0e", "0e", 3000, 16, 16, 16)])
def test_against_the_oracle(ir1, ir2, ir_out, n, c1, c2, c_out):
    g = torch.Generator().manual_seed(n)
    layer = enn.TensorProduct(ir1, ir2, ir_out, c1, c2, c_out, internal_weights=False, feature_mode="uvw").to(DEV)
    x1, x2 = torch.randn(n, layer.irreps_in1_dim, c1, generator=g), torch.randn(n, layer.irreps_in2_dim, c2, generator=g)
    w, cot = torch.randn(*layer.weight_shape, generator=g), torch.randn(n, layer.irreps_out_dim, c_out, generator=g)
    leaves = [t.to(DEV).requires_grad_(True) for t in (x1, x2, w)]
    out = layer(*leaves)
    assert type(out.grad_fn).__name__ == TensorProductUVW.__name__ + "Backward"
    got = [out, *torch.autograd.grad(out, leaves, cot.to(DEV))]
    where = DEV if n > 1000 else "cpu"                                    # the oracle's float64 sums of large batches
    ref = [t.to(where).double().requires_grad_(True) for t in (x1, x2, w)]
    want = [otp.tensor_product_dense(*ref, layer.irreps_in1, layer.irreps_in2, layer.irreps_out, feature_mode="uvw")]
    want += torch.autograd.grad(want[0], ref, cot.to(where).double())
    # output and operand gradients: splits of both factors 2^-22 each and chains of at most 160 multiply-adds (0.4 x 2^-24 x sqrt(160 / 2): 2.1e-7
    # where all are as long); weights: chains of 80 multiply-adds below 512 samples and for 16 output channels (0.4 x 2^-24 x sqrt(80 / 2) and the roundings of the
    # product of three: 2e-7), else truncation by the tensor core, up to 24 steps between two folds
    for k, (a, b) in enumerate(zip(got, want)):
        assert _rel(a, b.cpu()) < (2.45e-7 if k < 3 else 2.5e-7 if n < 512 or c_out == 16 else 8e-7), k
    (only,) = torch.autograd.grad(layer(leaves[0].detach(), leaves[1], w.to(DEV)), [leaves[1]], cot.to(DEV))
    assert _rel(only, want[2].cpu()) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("ir,c,taken", [("2x0e+2x1o+2x2e", 16, True), ("3x2e", 16, True), ("6x2e", 16, False)])
def test_chains_of_many_paths(ir, c, taken):
    """Several paths between the same irreps lengthen the sums of an output element: they are cut at 160 terms, and a layer whose paths do
    not fit that for the channels of one accumulator runs the composed products."""
    g = torch.Generator().manual_seed(5)
    n = 2500
    layer = enn.TensorProduct(ir, ir, ir, c, c, c, internal_weights=False, feature_mode="uvw").to(DEV)
    x1, x2 = torch.randn(n, layer.irreps_in1_dim, c, generator=g), torch.randn(n, layer.irreps_in2_dim, c, generator=g)
    w, cot = torch.randn(*layer.weight_shape, generator=g), torch.randn(n, layer.irreps_out_dim, c, generator=g)
    leaves = [t.to(DEV).requires_grad_(True) for t in (x1, x2, w)]
    out = layer(*leaves)
    assert (type(out.grad_fn).__name__ == TensorProductUVW.__name__ + "Backward") == taken
    got = [out, *torch.autograd.grad(out, leaves, cot.to(DEV))]
    ref = [t.to(DEV).double().requires_grad_(True) for t in (x1, x2, w)]
    want = [otp.tensor_product_dense(*ref, layer.irreps_in1, layer.irreps_in2, layer.irreps_out, feature_mode="uvw")]
    want += torch.autograd.grad(want[0], ref, cot.to(DEV).double())
    for a, b in zip(got[:3] if taken else got, want):
        assert _rel(a, b.cpu()) < (2.45e-7 if taken else 5e-6)      # 5e-6: sums of 4096 terms and more in one float32 chain
    if taken:
        assert _rel(got[3], want[3].cpu()) < 2.5e-7


@pytest.mark.gpu
def test_second_derivatives_are_those_of_the_composed_product():
    g = torch.Generator(device=DEV).manual_seed(3)
    ir, c, n = "0e+1o+2e", 16, 70
    layer = enn.TensorProduct(ir, ir, ir, c, c, c, internal_weights=False, feature_mode="uvw").to(DEV)
    leaves = [torch.randn(*s, generator=g, device=DEV).requires_grad_(True) for s in ((n, 9, c), (n, 9, c), layer.weight_shape)]
    cot = torch.randn(n, 9, c, generator=g, device=DEV)
    results = []
    for fn in (layer, lambda *a: tensor_product_uvw(*a, layer.tp_info_forward, layer.tp_info_backward1, layer.tp_info_backward2)):
        first = torch.autograd.grad(fn(*leaves), leaves, cot, create_graph=True)
        results.append([*first, *torch.autograd.grad(sum(t.square().sum() for t in first), leaves)])
    for a, b in zip(*results):
        assert _rel(a, b.cpu()) < 1e-5


def _peak(call):
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    result = call()
    torch.cuda.synchronize()
    return torch.cuda.max_memory_allocated() - base - sum(t.numel() * 4 for t in result), result


@pytest.mark.gpu
def test_scratch_stays_below_the_limit(monkeypatch):
    """Batches whose partial outputs would exceed the limit run in slices of whole sample tiles: forward and backward below it (the packed
    weights and the copies of the operands' gradients beside it), results as close to float64 as those of one call."""
    g = torch.Generator(device=DEV).manual_seed(7)
    ir, c, n = "2x0e+2x1o+2x2e", 16, 5003
    layer = enn.TensorProduct(ir, ir, ir, c, c, c, internal_weights=False, feature_mode="uvw").to(DEV)
    x1, x2, cot = (torch.randn(n, 18, c, generator=g, device=DEV) for _ in range(3))
    w = torch.randn(*layer.weight_shape, generator=g, device=DEV)
    leaves = [t.requires_grad_(True) for t in (x1, x2, w)]

    def call():
        out = layer(*leaves)
        return [out, *torch.autograd.grad(out, leaves, cot)]
    whole_peak, _ = _peak(call)
    limit = 16 << 20
    monkeypatch.setattr(ftp, "UVW_INTERMEDIATE_LIMIT", limit)
    peak, got = _peak(call)
    assert whole_peak > 2 * limit and peak < 1.5 * limit
    ref = [t.detach().double().requires_grad_(True) for t in leaves]
    want = [otp.tensor_product_dense(*ref, layer.irreps_in1, layer.irreps_in2, layer.irreps_out, feature_mode="uvw")]
    want += torch.autograd.grad(want[0], ref, cot.double())
    for a, b in zip(got, want):
        assert _rel(a, b.cpu()) < 2.5e-7


@pytest.mark.gpu
def test_differentiable_weight_gradient_stays_below_the_limit(monkeypatch):
    """A weight gradient that is to be differentiated again keeps no intermediate of the whole batch, and its derivatives are those of
    the product; a gradient that does not lie on 16 bytes takes the same kernels as one that does."""
    g = torch.Generator(device=DEV).manual_seed(9)
    ir, c, n = "0e+1o+2e", 16, 4000
    layer = enn.TensorProduct(ir, ir, ir, c, c, c, internal_weights=False, feature_mode="uvw").to(DEV)
    leaves = [torch.randn(*s, generator=g, device=DEV).requires_grad_(True) for s in ((n, 9, c), (n, 9, c), layer.weight_shape)]
    cot, v = torch.randn(n, 9, c, generator=g, device=DEV).requires_grad_(True), torch.randn(*layer.weight_shape, generator=g, device=DEV)
    out = layer(*leaves)

    def call():
        return list(torch.autograd.grad(out, leaves[2:], cot, create_graph=True, retain_graph=True))
    limit = 16 << 20                                        # the intermediate of the whole batch: 143 MB
    monkeypatch.setattr(ftp, "UVW_INTERMEDIATE_LIMIT", limit)
    peak, (gw,) = _peak(call)
    assert peak < 3 * limit
    got = [gw, *torch.autograd.grad(gw, [leaves[0], leaves[1], cot], v)]
    ref = [t.detach().double().requires_grad_(True) for t in (*leaves, cot)]
    dense = otp.tensor_product_dense(*ref[:3], layer.irreps_in1, layer.irreps_in2, layer.irreps_out, feature_mode="uvw")
    (want,) = torch.autograd.grad(dense, ref[2:3], ref[3], create_graph=True)
    for a, b in zip(got, [want, *torch.autograd.grad(want, [ref[0], ref[1], ref[3]], v.double())]):
        assert _rel(a, b.cpu()) < 3e-6                     # sums of 256 terms and of 4000 samples in two steps

    shifted = torch.empty(n * 9 * c + 1, device=DEV)[1:].view(n, 9, c).copy_(cot.detach())
    assert shifted.data_ptr() % 16 == 4
    for a, b in zip(torch.autograd.grad(out, leaves, shifted, retain_graph=True), torch.autograd.grad(out, leaves, cot.detach())):
        assert torch.equal(a, b)

