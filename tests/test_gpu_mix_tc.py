"""Tensor-core (tcgen05, 3xTF32) weight step against the CUDA-core kernel and a float64 einsum."""
import pytest
import torch

from equitorch_b200 import nn as enn
from equitorch_b200.irreps import Irreps
from equitorch_b200.ops import batched_sparse_dense_op as gops
from equitorch_b200.ops.fused_tp_op import check_status
from equitorch_b200.ops.mix_tc_op import MixPlan, mix_tc, mix_tc_transposed, wgrad_tc
from equitorch_b200.tables import tp_infos

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("irreps,n,cin,cout", [
    ("0e+1o+2e+3o", 1000, 64, 64), ("0e+1o+2e+3o", 37, 64, 64), ("0e+1o+2e", 513, 32, 48),
    ("0e+1o+2e+3o", 20011, 64, 64), ("2x0e+1o", 300, 64, 128),
])
def test_mix_tc_matches_float64(irreps, n, cin, cout):
    ir = Irreps(irreps)
    fwd, _, _, paths = tp_infos(ir, ir, Irreps("0e+1o+2e+3o"))
    info = fwd.info_M_fwd.to(DEV)
    plan = MixPlan(info, [i.dim for i in ir], DEV)
    assert plan.regular
    g = torch.Generator().manual_seed(n)
    s = torch.randn(n, plan.rows, cin, generator=g).to(DEV)
    w = (torch.randn(paths, cin, cout, generator=g) / cin ** 0.5).to(DEV)
    got = mix_tc(s, w, plan)
    check_status()
    simt = gops.indexed_vecmat_scale_gather(s, w, None, None, info.index2, info.seg_out, out_size=info.out_size)
    sel = w.double()[info.index2]                                    # (rows, cin, cout)
    per_row = torch.einsum("nri,rio->nro", s.double(), sel)
    seg = info.seg_out.cpu() if info.seg_out is not None else torch.arange(info.out_size + 1)
    want = torch.stack([per_row[:, seg[m]:seg[m + 1]].sum(1) for m in range(info.out_size)], 1)
    scale = float(want.abs().max())
    err_tc = float((got.double() - want).abs().max()) / scale
    err_simt = float((simt.double() - want).abs().max()) / scale
    # the float32 accumulation inside the tensor core is not round-to-nearest: a few 1e-6 of the largest
    # element is what the hardware gives; the parity bar for float32 results is 1e-5
    assert err_tc < 8e-6, f"tensor-core path: relative error {err_tc:.2e} (CUDA-core path {err_simt:.2e})"


@pytest.mark.parametrize("irreps,n,cin,cout", [("0e+1o+2e+3o", 1000, 64, 64), ("0e+1o+2e", 77, 48, 32),
                                               ("0e+1o+2e+3o", 20011, 64, 64)])
def test_mix_tc_transposed_is_the_adjoint(irreps, n, cin, cout):
    ir = Irreps(irreps)
    fwd, _, _, paths = tp_infos(ir, ir, Irreps("0e+1o+2e+3o"))
    info = fwd.info_M_fwd.to(DEV)
    plan = MixPlan(info, [i.dim for i in ir], DEV)
    gen = torch.Generator().manual_seed(n + 1)
    g = torch.randn(n, plan.comps, cout, generator=gen).to(DEV)
    w = (torch.randn(paths, cin, cout, generator=gen) / cout ** 0.5).to(DEV)
    got = mix_tc_transposed(g, w, plan)
    check_status()
    seg = info.seg_out.cpu() if info.seg_out is not None else torch.arange(info.out_size + 1)
    comp_of_row = torch.repeat_interleave(torch.arange(info.out_size), seg[1:] - seg[:-1]).to(DEV)
    want = torch.einsum("nro,rio->nri", g.double()[:, comp_of_row], w.double()[info.index2])
    err = float((got.double() - want).abs().max() / want.abs().max())
    assert got.shape == want.shape and err < 8e-6, f"relative error {err:.2e}"


@pytest.mark.parametrize("irreps,n,cin,cout", [("0e+1o+2e+3o", 1000, 64, 64), ("0e+1o+2e", 77, 32, 32),
                                               ("0e+1o+2e+3o", 20011, 64, 64), ("0e+1o+2e+3o", 5, 64, 64)])
def test_wgrad_tc_matches_float64_and_is_reproducible(irreps, n, cin, cout):
    ir = Irreps(irreps)
    fwd, _, _, paths = tp_infos(ir, ir, Irreps("0e+1o+2e+3o"))
    info = fwd.info_M_fwd.to(DEV)
    plan = MixPlan(info, [i.dim for i in ir], DEV)
    gen = torch.Generator().manual_seed(n + 2)
    s = torch.randn(n, plan.rows, cin, generator=gen).to(DEV)
    g = torch.randn(n, plan.comps, cout, generator=gen).to(DEV)
    got = wgrad_tc(s, g, plan, paths)
    again = wgrad_tc(s, g, plan, paths)
    check_status()
    assert torch.equal(got, again)
    seg = info.seg_out.cpu() if info.seg_out is not None else torch.arange(info.out_size + 1)
    comp_of_row = torch.repeat_interleave(torch.arange(info.out_size), seg[1:] - seg[:-1]).to(DEV)
    per_row = torch.einsum("nri,nro->rio", s.double(), g.double()[:, comp_of_row])
    want = torch.zeros(paths, cin, cout, dtype=torch.float64, device=DEV).index_add_(0, info.index2, per_row)
    err = float((got.double() - want).abs().max() / want.abs().max())
    assert err < 8e-6, f"relative error {err:.2e}"


@pytest.mark.parametrize("cout", [96, 128])
def test_sums_run_in_the_order_of_the_channels(cout):
    """One issuer (more than 64 columns): terms of one accumulator are added in the order of the channels, eight at a time.  2^30 + 1 is
    not a float32, so what cancels 2^30 in the last eight leaves 0, and 1 where the 1 comes after it."""
    ir = Irreps("2x0e+1o")
    fwd, _, _, paths = tp_infos(ir, ir, ir)
    plan = MixPlan(fwd.info_M_fwd.to(DEV), [i.dim for i in ir], DEV)
    s, w = torch.zeros(200, plan.rows, 32, device=DEV), torch.ones(paths, 32, cout, device=DEV)
    for place, value in ((0, 2. ** 30), (16, 1.), (24, -2. ** 30)):
        s[:, 0, place] = value
    got = mix_tc(s, w, plan)
    check_status()
    assert torch.count_nonzero(got) == 0


@pytest.mark.parametrize("bits", [0x7fffffff, -1, 0x7fc00000, 0x7f800001, 0x7f800000])
@pytest.mark.parametrize("c,cout", [(32, 32), (64, 64), (64, 128)])
def test_values_that_are_not_finite_reach_what_they_enter(bits, c, cout):
    """The pair of TF32 values of an operand is made in integer arithmetic, in which the largest NaNs wrap around."""
    g = torch.Generator().manual_seed(5)
    n = 700
    layer = enn.IrrepsLinear("0e+1o", "0e+1o", c, cout, internal_weights=False).to(DEV)
    x = torch.randn(n, 4, c, generator=g)
    x.view(torch.int32)[13, 2, 3] = bits
    w = torch.randn(*layer.weight_shape, generator=g)
    xg, wg = x.to(DEV).requires_grad_(), w.to(DEV).requires_grad_()
    out = layer(xg, wg)
    (gw,) = torch.autograd.grad(out, wg, torch.randn(n, 4, cout, generator=g).to(DEV))
    bad = torch.zeros(n, 4, cout, dtype=torch.bool, device=DEV)
    bad[13, 2] = True
    assert torch.equal(~torch.isfinite(out), bad)
    worse = torch.zeros(gw.shape, dtype=torch.bool, device=DEV)
    worse[1, 3] = True                                  # the row of 1o that the value is a factor of
    assert torch.equal(~torch.isfinite(gw), worse)


# one node; a tile of 40 rows and one more; fewer tiles than CTAs; chunks of eight tiles and their remainders.  Irreps that fill a tile of 40
# rows, leave padding, or are longer than one (41: one node a tile; 65: one issuer and two slots at 64 columns)
@pytest.mark.parametrize("irreps", ["0e+1o+2e+3o", "9o+10e", "20e+0e", "32e+1o"])
@pytest.mark.parametrize("n,cin,cout", [(1, 32, 32), (40, 64, 64), (41, 32, 96), (333, 96, 64), (2600, 64, 128), (9001, 32, 64)])
def test_wgrad_tc_at_the_edges_of_its_tiles(irreps, n, cin, cout):
    if irreps == "32e+1o" and cout > 64:
        pytest.skip("an irrep of 65 components does not fit beside more than 64 columns")
    ir = Irreps(irreps)
    fwd, _, _, paths = tp_infos(ir, ir, Irreps("0e"))
    info = fwd.info_M_fwd.to(DEV)
    plan = MixPlan(info, [i.dim for i in ir], DEV)
    gen = torch.Generator().manual_seed(n + cout)
    s = torch.randn(n, plan.rows, cin, generator=gen).to(DEV)
    g = torch.randn(n, plan.comps, cout, generator=gen).to(DEV)
    got = wgrad_tc(s, g, plan, paths)
    check_status()
    seg = info.seg_out.cpu() if info.seg_out is not None else torch.arange(info.out_size + 1)
    comp_of_row = torch.repeat_interleave(torch.arange(info.out_size), seg[1:] - seg[:-1]).to(DEV)
    want = torch.zeros(paths, cin, cout, dtype=torch.float64, device=DEV)
    for r in range(plan.rows):
        want[int(info.index2[r])] += s[:, r].double().T @ g[:, int(comp_of_row[r])].double()
    assert float((got.double() - want).abs().max()) <= 8e-6 * float(want.abs().max())


# one, two, four and more splits of a block, whose sums one, two, four and eight warps add up; one issuer (more than 64 columns) with one to
# six tiles a CTA, folded in thirds.  A part of K terms of random sign added by rounding halves, or by truncation in the tensor core, whose
# steps of eight terms are off by up to a unit each, stays below 2^-24 (sqrt(K / 6) + K / 24); parts are at most 96 terms and the CTAs' sums
# of K' parts add sqrt(K' / 6), here below 4; the operands' pairs of TF32 values leave 2^-22.
@pytest.mark.parametrize("n", [1, 5, 20, 33, 60, 130, 1500])
@pytest.mark.parametrize("irreps,cin,cout", [("3o", 64, 64), ("0e+1o+2e+3o+4e", 128, 128), ("3x1o", 32, 96)])
def test_weight_gradient_of_few_nodes(irreps, cin, cout, n):
    ir = Irreps(irreps)
    fwd, _, _, paths = tp_infos(ir, Irreps("0e"), ir)
    info = fwd.info_M_fwd.to(DEV)
    plan = MixPlan(info, [i.dim for i in ir], DEV)
    gen = torch.Generator().manual_seed(n)
    s, g = torch.randn(n, plan.rows, cin, generator=gen).to(DEV), torch.randn(n, plan.comps, cout, generator=gen).to(DEV)
    got = wgrad_tc(s, g, plan, paths)
    check_status()
    seg = info.seg_out.cpu() if info.seg_out is not None else torch.arange(info.out_size + 1)
    comp_of_row = torch.repeat_interleave(torch.arange(info.out_size), seg[1:] - seg[:-1]).to(DEV)
    path_of_row = info.index2 if info.index2 is not None else torch.arange(plan.rows, device=DEV)
    per_row = torch.einsum("nri,nro->rio", s.double(), g.double()[:, comp_of_row])
    want = torch.zeros(paths, cin, cout, dtype=torch.float64, device=DEV).index_add_(0, path_of_row, per_row)
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -24 * (4 + 4 + 4) + 2.0 ** -22
