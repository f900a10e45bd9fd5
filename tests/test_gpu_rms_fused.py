"""One-pass gate gradients, training-mode BatchRMSNorm and register-resident LayerRMSNorm against plain float64 torch, at the
sizes where their tiles end: one sample, fewer rows than a block's pass, rows longer than a block, odd channel counts."""
import pytest
import torch

from equitorch_b200 import nn as enn
from equitorch_b200.irreps import Irreps
from equitorch_b200.tables import irreps_info
from oracle import norm_gate as ong

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# (irreps, channels): 1-vector rows, 65 vectors (odd, above two per lane), the 8-vector instance, 784 vectors (two column
# tiles, above the register rows), 5 channels (no vectors at all)
SHAPES = [("0e", 4), ("0e+1o+2e", 32), ("4x0e+2x1o+2e", 64), ("0e+1o+2e+3o", 64), ("0e+1o+2e+3o", 128),
          ("0e+1o+2e+3o+4e+5o+6e", 64), ("0e+1o", 5)]
SIZES = [1, 2, 37, 3001]


def _info(ir, dtype):
    """The tables with their 1 / dim factors in the features' precision."""
    info = irreps_info(ir).to(DEV)
    dims = torch.tensor([i.dim for i in ir], dtype=dtype, device=DEV)
    return info._replace(rdims=1 / dims, rsqrt_dims=dims.rsqrt())


def _inputs(ir, n, c, dtype):
    g = torch.Generator().manual_seed(n * 131 + c)
    make = lambda *shape: torch.randn(*shape, generator=g, dtype=torch.float64).to(dtype)
    return make(n, ir.dim, c), make(n, len(ir), c), make(len(ir), c) * 0.2 + 1, make(n, ir.dim, c)


def _close(got, want, tol, terms=0.0):
    """Largest difference over the largest value; ``terms`` is the size of the first of the two terms that the gradient of the
    features is the difference of (for one sample and one component they cancel, and rounding is relative to them)."""
    for i, (a, b) in enumerate(zip(got, want)):
        assert a.shape == b.shape
        size = max(float(b.detach().abs().max()), terms if i == 1 else 0.0)
        assert float((a.detach().double().cpu() - b.detach()).abs().max()) <= tol * size


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float64, 1e-12)])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("name,c", SHAPES)
def test_chain_matches_float64(name, c, n, dtype, tol):
    ir = Irreps(name)
    dims = [i.dim for i in ir]
    x, s, w, cot = _inputs(ir, n, c, dtype)
    bn, ln, gate = enn.BatchRMSNorm(ir, c), enn.LayerRMSNorm(ir, c), enn.Gate(ir)
    for m in (bn, ln, gate):
        m.to(DEV, dtype).train()
        m.irreps_info = _info(ir, dtype)
    for m in (bn, ln):
        m.weight = torch.nn.Parameter(w.to(DEV))
    xg, sg = (t.to(DEV).requires_grad_(True) for t in (x, s))
    term = lambda out: float((cot.double() * out / xo).detach().abs().max())
    xo, so, wb, wl = (t.double().requires_grad_(True) for t in (x, s, w, w))
    run0 = torch.ones(len(ir), c, dtype=torch.float64)
    ref_bn, run = ong.batch_rms_norm(xo, run0, dims, wb, True, True, 0.1, 1e-5)
    want_bn = [ref_bn, *torch.autograd.grad(ref_bn, [xo, wb], cot.double()), run]
    got_bn = bn(xg)
    _close([got_bn, *torch.autograd.grad(got_bn, [xg, bn.weight], cot.to(DEV)), bn.running_squared_norm], want_bn, tol, term(ref_bn))
    ref_ln, ref_gate = ong.layer_rms_norm(xo, dims, wl, True, 1e-5), ong.gate(xo, so, dims, None)
    got_ln, got_gate = ln(xg), gate(xg, sg)
    _close([got_ln, *torch.autograd.grad(got_ln, [xg, ln.weight], cot.to(DEV))],
           [ref_ln, *torch.autograd.grad(ref_ln, [xo, wl], cot.double())], tol, term(ref_ln))
    _close([got_gate, *torch.autograd.grad(got_gate, [xg, sg], cot.to(DEV))],
           [ref_gate, *torch.autograd.grad(ref_gate, [xo, so], cot.double())], tol)


@pytest.mark.parametrize("affine,scaled", [(True, True), (False, True), (True, False)])
def test_batch_norm_and_gate_second_derivatives(affine, scaled):
    ir, c, n = Irreps("0e+1o+2e"), 4, 5
    x, s, w, _ = _inputs(ir, n, c, torch.float64)
    bn = enn.BatchRMSNorm(ir, c, affine=affine, scaled=scaled).to(DEV).double().train()
    bn.irreps_info = _info(ir, torch.float64)
    gate = enn.Gate(ir).to(DEV)
    params = [x.to(DEV).requires_grad_(True), s.to(DEV).requires_grad_(True)]

    def chain(a, b):
        return bn(gate(a, b))

    assert torch.autograd.gradcheck(chain, params)
    assert torch.autograd.gradgradcheck(chain, params)


def test_transposed_gradient_and_features():
    """A gradient and features that are views with other strides give what their copies give."""
    ir, c, n = Irreps("0e+1o+2e"), 32, 65
    x, s, w, cot = (t.to(DEV) for t in _inputs(ir, n, c, torch.float32))
    bn, gate = enn.BatchRMSNorm(ir, c).to(DEV).train(), enn.Gate(ir).to(DEV)
    results = []
    for view in (False, True):
        a, b = ((t.transpose(0, 2).contiguous().transpose(0, 2) if view else t) for t in (x, cot))
        a = a.detach().requires_grad_(True)
        sg = s.clone().requires_grad_(True)
        out = bn(gate(a, sg))
        results.append([out, *torch.autograd.grad(out, [a, sg, bn.weight], b)])
    for p, q in zip(*results):
        assert torch.equal(p, q)


def test_weights_that_broadcast_are_taken_as_before():
    from equitorch_b200.nn import functional as F
    ir, c, n = Irreps("0e+1o+2e"), 8, 11
    x, _, w, _ = (t.to(DEV) for t in _inputs(ir, n, c, torch.float32))
    info = _info(ir, torch.float32)
    for weight in (w[:, :1], w[:1], w[0]):
        a, b = torch.ones(len(ir), c, device=DEV), torch.ones(len(ir), c, device=DEV)
        got = F.batch_rms_norm(x, a, info, weight, True, True, 0.1, 1e-5)
        want = F.batch_rms_norm(x, b, info, weight.expand(len(ir), c), True, True, 0.1, 1e-5)
        assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max()) and torch.allclose(a, b, rtol=1e-5)


@pytest.mark.parametrize("ir,n,c", [("0e+1o+2e+3o", 20000, 64), ("0e+1o+2e", 5000, 64), ("0e+1o", 700, 32)])
def test_normalisations_are_no_further_from_64_bits(ir, n, c):
    """2-norm errors of outputs and gradients, over the norms, against those of the per-irrep operators they replace (batch: 5.4e-8,
    6.0e-8, 1.16e-7 or more; layer: 5.8e-8, 5.9e-8, 1.3e-7 or more); a tenth for other draws."""
    from equitorch_b200 import nn as enn
    g = torch.Generator().manual_seed(n)
    for cls, bounds in ((enn.BatchRMSNorm, (5.4e-8, 6.0e-8, 1.16e-7)), (enn.LayerRMSNorm, (5.8e-8, 6.0e-8, 1.3e-7))):
        layer = cls(ir, c)
        dim, weight = layer.irreps.dim, torch.randn(*layer.weight.shape, generator=g)
        x, cot = torch.randn(n, dim, c, generator=g), torch.randn(n, dim, c, generator=g)
        results = []
        for dtype in (torch.float32, torch.float64):
            torch.set_default_dtype(dtype)
            try:
                m = cls(ir, c).to("cuda:0")
            finally:
                torch.set_default_dtype(torch.float32)
            m.weight.data.copy_(weight)
            leaf = x.to(dtype).to("cuda:0").requires_grad_(True)
            out = m(leaf)
            results.append([out.detach(), *torch.autograd.grad(out, [leaf, m.weight], cot.to(dtype).to("cuda:0"))])
        for a, b, bound in zip(*results, bounds):
            assert float((a.double() - b).norm() / b.norm()) < 1.1 * bound
