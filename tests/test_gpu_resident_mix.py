"""``IrrepsLinear`` on the tensor-core product that keeps an output row's weights in shared memory, against float64: widths of one and
of two accumulator units, sums of one to four k-blocks (the most it takes), batches that end inside a sample tile, ranges that begin and
end inside an output row, a row that no path reaches, and rows that several outputs read; and the calls that the kernel with a
ring of weights keeps (narrow outputs, fewer items than SMs, longer sums)."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from equitorch_b200 import _lib
from equitorch_b200 import nn as enn
from equitorch_b200.ops import indexed_tc_op as tc
from equitorch_b200.ops.fused_tp_op import check_status, status_flag

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("ir_in,ir_out,n,cin,cout,passes", [
    ("0e+1o+2e+3o", "0e+1o+2e+3o", 4003, 64, 128, 2), ("0e+1o", "0e+1o", 20011, 32, 128, 1), ("0e+1o+2e", "0e+1o+2e", 2100, 64, 48, 1),
    ("0e+1o", "0e+1o", 5003, 128, 64, 1), ("0e+1o+2e", "0e+1o+2e", 2500, 96, 16, 0), ("0e+1o", "0e+1o", 6400, 160, 32, 0),
    ("0e+1o", "0e+1e+1o", 5003, 64, 64, 1), ("0e+1o", "2x0e+2x1o", 5003, 64, 64, 1), ("2x0e+1o", "0e+1o", 5003, 64, 128, 1),
    ("0e", "0e", 19000, 96, 64, 1), ("0e+1o+2e+3o", "0e+1o+2e+3o", 4003, 64, 64, 2),
    ("0e+1o+2e+3o", "0e+1o+2e+3o", 513, 64, 128, 0), ("0e+1o", "0e+1o", 700, 32, 64, 0), ("0e", "0e", 512, 128, 128, 0)])
def test_against_float64(ir_in, ir_out, n, cin, cout, passes):
    """``passes``: how many of the two products (output, gradient of x) take the resident kernel."""
    g = torch.Generator(device=DEV).manual_seed(n)
    layer = enn.IrrepsLinear(ir_in, ir_out, cin, cout, internal_weights=False).to(DEV)
    x = torch.randn(n, layer.irreps_in.dim, cin, generator=g, device=DEV).requires_grad_(True)
    w = (torch.randn(*layer.weight_shape, generator=g, device=DEV) * cin ** -0.5).requires_grad_(True)
    cot = torch.randn(n, layer.irreps_out.dim, cout, generator=g, device=DEV)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = layer(x, w)
        got = [out, *torch.autograd.grad(out, [x, w], cot)]
        check_status(torch.device(DEV))
    assert sum(e.count for e in prof.key_averages() if "vecmat_resident_kernel" in e.key) == passes
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    f = layer.forward_info
    want = xd.new_zeros(n, layer.irreps_out.dim, cout)
    seg = f.M_seg_MM0.tolist()
    rows = []
    for r in range(len(seg) - 1):
        rows.append(sum(f.scale_MM0[t].double() * xd[:, f.M0_MM0[t]] @ wd[f.ii0_MM0[t]] for t in range(seg[r], seg[r + 1])))
    want = want.index_add(1, f.M_out, torch.stack(rows, dim=1))
    # three products of TF32 pairs, at most eight truncating steps per accumulator: a few units of 2^-24
    for a, b in zip(got, [want, *torch.autograd.grad(want, [xd, wd], cot.double())]):
        assert _rel(a.detach(), b.detach()) < 2e-6


def test_groups_longer_than_announced_are_reported():
    """The buffers are sized by the caller's ``longest``: a group past it must end in an error, not past the buffers."""
    n, cin, cout, dim = 20000, 128, 64, 4
    x, w = torch.randn(n, dim, cin, device=DEV), torch.randn(dim, cin, cout, device=DEV)
    index = torch.arange(dim, device=DEV)
    plan = tc.VecmatPlan(index, None, dim, dim, cin, cout, torch.device(DEV))
    assert plan.group == 1 and plan.longest == 4
    want = tc.vecmat_tc(x, w, None, index, index, None, dim)
    plan.longest = 1
    packed, out = torch.empty(2, dim * cin * cout, device=DEV), torch.empty(n, dim, cout, device=DEV)

    def call():
        _lib.check(_lib.lib().eqt_vecmat_tc_grouped(
            x.data_ptr(), w.data_ptr(), index.data_ptr(), None, packed[0].data_ptr(), packed[1].data_ptr(), out.data_ptr(), n, dim, cin,
            cout, dim, plan.slots, plan.group, plan.num_groups, plan.group_rows.data_ptr(), plan.slot_entry.data_ptr(),
            plan.kb_begin.data_ptr(), plan.a_col.data_ptr(), plan.longest, status_flag(x.device).data_ptr(), _lib.stream_ptr(x.device)), "call")
    call()
    with pytest.raises(_lib.EqtError, match="longer than"):
        check_status(x.device)
    plan.longest = 4
    call()
    check_status(x.device)
    assert torch.equal(out, want)
