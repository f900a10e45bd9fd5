"""The tensor-core paths behind ``indexed_vecmat_scale_gather`` (shared matrix operand) and accumulated
``indexed_outer_scale_gather``: against the float64 oracle and against the table-driven CUDA-core kernels, on random
tables with empty segments, missing index arrays and ragged batch sizes; and the layers that reach them through
the reference's own entry points (IrrepWiseLinear, IrrepsLinear, SO2Linear, per-edge SO3Linear 'uv').
Error norm: max |a - b| / max |b|, bound 1e-5 (float32, 3xTF32 products with float32 accumulation)."""
import pytest
import torch

from equitorch_b200 import nn as enn
from equitorch_b200.ops import batched_sparse_dense_op as gops
from equitorch_b200.ops import indexed_tc_op as tc
from equitorch_b200.ops.fused_tp_op import check_status
from oracle import sparse_ops as oops
from oracle import tensor_products as otp

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rel(a, b):
    return float((a.detach().double().cpu() - b.detach().double().cpu()).abs().max() / max(1e-30, float(b.detach().abs().max())))


def _table(g, entries, rows1, rows2, num_out, with_index1=True, with_index2=True, with_scale=True):
    # sorted output rows with some empty segments
    owner = torch.sort(torch.randint(0, num_out, (entries,), generator=g)).values
    owner = owner[owner != num_out // 2] if num_out > 2 else owner          # one row without entries
    entries = owner.numel()
    seg = torch.zeros(num_out + 1, dtype=torch.long)
    seg[1:] = torch.cumsum(torch.bincount(owner, minlength=num_out), 0)
    i1 = torch.randint(0, rows1, (entries,), generator=g) if with_index1 else None
    i2 = torch.randint(0, rows2, (entries,), generator=g) if with_index2 else None
    sc = torch.randn(entries, generator=g) if with_scale else None
    return sc, i1, i2, seg, entries


@pytest.mark.parametrize("n,cin,cout", [(1000, 32, 32), (777, 64, 48), (4096, 32, 64), (513, 96, 128)])
@pytest.mark.parametrize("variant", ["full", "no_index2", "no_scale"])
def test_vecmat_shared_weights(n, cin, cout, variant):
    g = torch.Generator().manual_seed(n + cin + cout)
    rows1, rows2, num_out = 13, 9, 11
    sc, i1, i2, seg, entries = _table(g, 40, rows1, rows2, num_out, with_index2=variant != "no_index2",
                                      with_scale=variant != "no_scale")
    if i2 is None:
        rows2 = entries
    x = torch.randn(n, rows1, cin, generator=g)
    w = torch.randn(rows2, cin, cout, generator=g) / cin ** 0.5
    want = oops.indexed_vecmat_scale_gather(x.double(), w.double(), sc if sc is None else sc.double(), i1, i2, seg)
    dev = lambda t: None if t is None else t.to(DEV)
    assert tc.vecmat_supported(x.to(DEV), w.to(DEV), None, None, False, num_out, num_out)
    got = gops.indexed_vecmat_scale_gather(x.to(DEV), w.to(DEV), dev(sc), dev(i1), dev(i2), dev(seg))
    check_status()
    assert got.shape == want.shape and _rel(got, want) < 1e-5
    assert torch.count_nonzero(got[:, num_out // 2]) == 0                       # the row without entries
    # operands swapped: the matrix-transposed-vector alias reaches the same kernel
    got2 = gops.indexed_mat_t_vec_scale_gather(w.to(DEV), x.to(DEV), dev(sc), dev(i2), dev(i1), dev(seg))
    assert torch.equal(got, got2)


@pytest.mark.parametrize("n,c1,c2", [(1000, 32, 32), (999, 64, 32), (5000, 32, 64), (640, 64, 128)])
@pytest.mark.parametrize("variant", ["full", "no_scale"])
def test_outer_accumulated(n, c1, c2, variant):
    g = torch.Generator().manual_seed(n + c1 + c2)
    rows1, rows2, num_w = 7, 5, 9
    sc, i1, i2, seg, entries = _table(g, 30, rows1, rows2, num_w, with_scale=variant != "no_scale")
    a, b = torch.randn(n, rows1, c1, generator=g), torch.randn(n, rows2, c2, generator=g)
    want = oops.indexed_outer_scale_gather(a.double(), b.double(), sc if sc is None else sc.double(), i1, i2, seg,
                                           out_accumulated=True)
    dev = lambda t: None if t is None else t.to(DEV)
    assert tc.outer_supported(a.to(DEV), b.to(DEV), None, None, True, num_w, num_w)
    got = gops.indexed_outer_scale_gather(a.to(DEV), b.to(DEV), dev(sc), dev(i1), dev(i2), dev(seg), out_accumulated=True)
    again = gops.indexed_outer_scale_gather(a.to(DEV), b.to(DEV), dev(sc), dev(i1), dev(i2), dev(seg), out_accumulated=True)
    check_status()
    assert got.shape == want.shape and _rel(got, want) < 1e-5
    assert torch.equal(got, again)                                              # fixed summation order
    assert torch.count_nonzero(got[num_w // 2]) == 0


def test_layers_reach_tensor_cores_and_match_table_driven_kernels(monkeypatch):
    """IrrepWiseLinear, IrrepsLinear, SO2Linear and the per-edge SO3Linear 'uv' at 4096 samples: output and all
    gradients through the tensor-core paths against the same layers on the table-driven kernels (1e-5) and the
    number of tensor-core launches."""
    from equitorch_b200 import _lib
    g = torch.Generator().manual_seed(1)
    n, c = 4096, 32
    cases = [
        ("irrepwise", enn.IrrepWiseLinear("0e+1o+2e", c, c, internal_weights=False), 9),
        ("irreps", enn.IrrepsLinear("0e+1o+2e", "0e+1o+1o+2e", c, c, internal_weights=False), 9),
        ("so2", enn.SO2Linear("0e+1o+2e+3o", "0e+1o+2e+3o", c, c, internal_weights=False, feature_mode="uv"), 16),
    ]
    for name, layer, dim in cases:
        layer = layer.to(DEV)
        x = torch.randn(n, dim, c, generator=g).to(DEV).requires_grad_(True)
        w = (torch.randn(*layer.weight_shape, generator=g) / c ** 0.5).to(DEV).requires_grad_(True)
        out = layer(x, w)
        cot = torch.randn(out.shape, generator=g).to(DEV)
        grads = torch.autograd.grad(out, [x, w], cot)
        check_status()
        monkeypatch.setattr(tc, "MIN_BATCH", 1 << 60)                          # table-driven kernels
        ref = layer(x, w)
        ref_grads = torch.autograd.grad(ref, [x, w], cot)
        monkeypatch.setattr(tc, "MIN_BATCH", 512)
        for u, v in [(out, ref), *zip(grads, ref_grads)]:
            assert _rel(u, v) < 1e-5, name


@pytest.mark.parametrize("ir,c", [("0e+1o+2e", 32), ("0e+1o+2e+3o", 16), ("0e+1o", 48)])
def test_tensor_product_uvw_sliced_over_samples(monkeypatch, ir, c):
    """The composed 'uvw' product with the intermediate limit lowered so that the batch is processed in slices (three of 512 samples, and
    a remainder): output and all three gradients against the float64 oracle (dense path form) on all samples and against
    the unsliced chain; bound 1e-5.  48 channels and l_max 3 take it from the layer as well."""
    from equitorch_b200.nn.functional import tensor_products as ftp
    n, dim = 1560, {"0e+1o": 4, "0e+1o+2e": 9, "0e+1o+2e+3o": 16}[ir]
    g = torch.Generator().manual_seed(2)
    layer = enn.TensorProduct(ir, ir, ir, c, c, c, internal_weights=False, feature_mode="uvw").to(DEV)
    infos = (layer.tp_info_forward, layer.tp_info_backward1, layer.tp_info_backward2)
    x1, x2 = torch.randn(n, dim, c, generator=g), torch.randn(n, dim, c, generator=g)
    w = torch.randn(*layer.weight_shape, generator=g) / c
    cot = torch.randn(n, dim, c, generator=g)
    leaves = [t.to(DEV).requires_grad_(True) for t in (x1, x2, w)]
    whole = ftp.tensor_product_uvw(*leaves, *infos)
    assert type(whole.grad_fn).__name__ == "TensorProductUVWDummyBackward"
    gwhole = torch.autograd.grad(whole, leaves, cot.to(DEV))
    monkeypatch.setattr(ftp, "UVW_INTERMEDIATE_LIMIT", 512 * infos[0].info_Mij_fwd.out_size * c * c * 4)       # slices of 512 samples
    sliced = (layer if (ir, c) != ("0e+1o+2e", 32) else lambda *a: ftp.tensor_product_uvw(*a, *infos))(*leaves)
    assert type(sliced.grad_fn).__name__ == "TensorProductUVWChunkedBackward"
    gsliced = torch.autograd.grad(sliced, leaves, cot.to(DEV))
    check_status()
    ref = [t.to(DEV).double().requires_grad_(True) for t in (x1, x2, w)]
    want = [otp.tensor_product_dense(*ref, ir, ir, ir, feature_mode="uvw")]
    want += torch.autograd.grad(want[0], ref, cot.to(DEV).double())
    for u, v, r in zip([sliced, *gsliced], [whole, *gwhole], want):
        assert _rel(u, v) < 1e-5 and _rel(u, r) < 1e-5


@pytest.mark.parametrize("which", ["indexed", "blocks"])
def test_weight_gradients_on_two_streams(which):
    """Two streams at once, each with its own inputs: every result is the one of the call alone (the partial sums of the
    split reduction belong to the call)."""
    from equitorch_b200.irreps import Irreps
    from equitorch_b200.ops.mix_tc_op import MixPlan, wgrad_tc
    from equitorch_b200.tables import tp_infos
    g = torch.Generator(device=DEV).manual_seed(0)
    n, c = 20000, 64
    ir = Irreps("0e+1o+2e")
    table, _, _, paths = tp_infos(ir, ir, ir)
    plan = MixPlan(table.info_M_fwd.to(DEV), [i.dim for i in ir], DEV)
    index, seg = torch.arange(9, device=DEV), torch.arange(10, device=DEV)
    inputs = [[torch.randn(n, rows, c, generator=g, device=DEV) for rows in ((9, 9) if which == "indexed" else (plan.rows, 9))] for _ in range(2)]

    def call(a, b):
        if which == "blocks":
            return wgrad_tc(a, b, plan, paths)
        return gops.indexed_outer_scale_gather(a, b, None, index, index, seg, out_accumulated=True)
    want = [call(*pair) for pair in inputs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(40):
        for k, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                got[k].append(call(*inputs[k]))
    torch.cuda.synchronize()
    for k in range(2):
        assert all(torch.equal(t, want[k]) for t in got[k])


def test_calls_that_can_have_no_plan_take_the_table_driven_kernels():
    """A first call while a stream is captured, and tables that belong to inference mode."""
    ir, n, c = "0e+1o+2e", 600, 32
    g = torch.Generator().manual_seed(3)
    x, w = torch.randn(n, 9, c, generator=g).to(DEV), torch.randn(3, c, c, generator=g).to(DEV)
    new = lambda: enn.IrrepsLinear(ir, ir, c, c, internal_weights=False).to(DEV)
    want = new()(x, w)
    layer, graph = new(), torch.cuda.CUDAGraph()
    with torch.no_grad():
        new()(x[:100], w)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            got = layer(x, w)
    graph.replay()
    torch.cuda.synchronize()
    assert _rel(got, want) < 1e-5
    with torch.inference_mode():
        assert _rel(new()(x, w).clone(), want) < 1e-5


@pytest.mark.parametrize("lmax,c", [(2, 32), (3, 64), (6, 32)])          # groups of 2 to 4 rows, some not full, of 64 to 128 columns
@pytest.mark.parametrize("n", [512, 513, 4999])                           # whole tiles of 128 samples, one sample more, several items a CTA
def test_rows_in_groups(lmax, c, n):
    import copy
    from equitorch_b200 import nn as enn
    from equitorch_b200.irreps import Irreps
    ir = Irreps((0, lmax))
    layer = enn.SO2Linear(ir, ir, c, c, internal_weights=False, feature_mode="uv").to(DEV)
    g = torch.Generator().manual_seed(n + lmax)
    x, cot = (torch.randn(n, ir.dim, c, generator=g).to(DEV) for _ in range(2))
    w = (torch.randn(*layer.weight_shape, generator=g) / c ** 0.5).to(DEV)
    results = []
    for module, dtype in ((layer, torch.float32), (copy.deepcopy(layer).double(), torch.float64)):
        xs, ws = x.to(dtype).requires_grad_(), w.to(dtype).requires_grad_()
        out = module(xs, ws)
        results.append([out, *torch.autograd.grad(out, [xs, ws], cot.to(dtype))])
    for got, want in zip(*results):
        assert float((got.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
