"""Segment sums and adjoints with one warp a node, or four where those are faster: rows, rows mixed channel by channel, and the
weights' gradient, against float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from equitorch_b200.irreps import Irreps
from equitorch_b200.ops.fused_tp_op import (INNER_CHANNELS, TpTable, cg_inner, cg_inner_mix, cg_segment_mix, cg_segment_sum,
                                            mix_scratch)
from equitorch_b200.tables import tp_infos

DEV = torch.device("cuda:0")
# float32 sums of at most a few hundred terms: 1e-5 of the largest entry, the path's tolerance
TOL = 1e-5


def _tables(lmax, role):
    ir = Irreps("+".join(f"{l}{'eo'[l % 2]}" for l in range(lmax + 1)))
    fwd, bwd1, _, _ = tp_infos(ir, ir, ir)
    info = fwd if role == "fwd" else bwd1
    table = TpTable(info.info_Mij_fwd, role == "fwd", ir.dim, ir.dim, DEV, info.info_M_fwd)
    row = torch.from_numpy(np.repeat(np.arange(table.num_rows), np.diff(table.row_ptr.cpu().numpy()))).to(DEV)
    m = info.info_M_fwd
    seg = m.seg_out.to(DEV)
    comp = torch.repeat_interleave(torch.arange(m.out_size, device=DEV), seg[1:] - seg[:-1])
    return ir.dim, table, row, comp, m.index2.to(DEV)


def _close(got, want):
    assert float((got.double() - want).abs().max()) <= TOL * max(float(want.abs().max()), 1e-30)


# one node of one edge; fewer nodes than warps; degrees over a ring, a block of 32 indices and its remainders, empty nodes in front and behind
DEGREES = {"one": [1], "few": [0, 3, 1, 0, 2, 5, 0], "blocks": [31, 32, 33, 0, 64, 65, 1, 4, 97], "many": None}


@pytest.mark.parametrize("degrees", list(DEGREES))
@pytest.mark.parametrize("c", [16, 32, 64, 96, 128])
@pytest.mark.parametrize("lmax,role", [(1, "fwd"), (1, "bwd1"), (2, "fwd"), (2, "bwd1"), (3, "fwd"), (3, "bwd1")])
def test_against_float64(lmax, role, c, degrees):
    dim, table, row, comp, path = _tables(lmax, role)
    g = torch.Generator().manual_seed(17 * lmax + c)
    deg = torch.tensor(DEGREES[degrees]) if DEGREES[degrees] else torch.randint(0, 7, (5003,), generator=g)
    n, e = deg.numel(), int(deg.sum())
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64), torch.cumsum(deg, 0)]).to(DEV)
    fidx, yidx = torch.randint(0, 50, (e,), generator=g).to(DEV), torch.randperm(e, generator=g).to(DEV)
    feat, y = torch.randn(50, dim, c, generator=g).to(DEV), torch.randn(e, dim, generator=g).to(DEV)
    x, w = torch.randn(n, dim, c, generator=g).to(DEV), torch.randn(int(path.max()) + 1, c, generator=g).to(DEV)
    grad = torch.randn(n, dim, c, generator=g).to(DEV)
    node = torch.repeat_interleave(torch.arange(n, device=DEV), deg.to(DEV))

    yd, sd = y.double()[yidx], table.scale.double()
    rows = torch.zeros(n, table.num_rows, c, dtype=torch.float64, device=DEV)
    gy = torch.zeros(e, dim, dtype=torch.float64, device=DEV)
    big = w.double()[path] * grad.double()[:, comp]                      # (n, rows, c): gradient of the rows
    for t0 in range(0, sd.numel(), 16):                                  # a few entries at a time: the terms of all would not fit
        t = slice(t0, t0 + 16)
        f = feat.double()[fidx][:, table.m_feat[t]] * sd[t, None]
        term = f * yd[:, table.m_y[t], None]
        rows.index_put_((node[:, None], row[None, t]), term, accumulate=True)
        gy.index_add_(1, table.m_y[t], (f * big[node][:, row[t]]).sum(-1))
    want = torch.zeros(n, dim, c, dtype=torch.float64, device=DEV).index_add_(1, comp, w.double()[path] * rows)
    gw = torch.zeros(w.shape, dtype=torch.float64, device=DEV).index_add_(0, path, (x.double()[:, comp] * rows).sum(0))
    want_gy = torch.zeros_like(gy)
    want_gy[yidx] = gy

    _close(cg_segment_sum(table, feat, y, fidx, yidx, ptr, n), rows)
    out, none = cg_segment_mix(table, feat, y, fidx, yidx, ptr, n, w)
    assert none is None
    _close(out, want)
    out, got_gw = cg_segment_mix(table, feat, y, fidx, yidx, ptr, n, w, x)
    _close(out, want)
    _close(got_gw, gw)
    _close(cg_inner(table, feat, big.float(), fidx, ptr, node, yidx, e), want_gy)
    if c in INNER_CHANNELS:
        _close(cg_inner_mix(table, feat, grad, w, fidx, ptr, yidx, e), want_gy)


# sums that four warps a node make because the rows that they write decide; from 100 nodes an SM on also the adjoint at l_max 3, 128 channels
@pytest.mark.parametrize("lmax,c,n", [(2, 128, 59_000), (3, 32, 38_500), (3, 64, 19_100), (3, 128, 14_900)])
def test_large_graphs_of_few_edges(lmax, c, n):
    dim, table, row, _, _ = _tables(lmax, "fwd")
    g = torch.Generator(device=DEV).manual_seed(n)
    e, some = 2 * n, torch.cat([torch.arange(200), torch.arange(n - 200, n)]).to(DEV)
    ptr, node = torch.arange(0, e + 1, 2, device=DEV), torch.arange(n, device=DEV).repeat_interleave(2)
    fidx = torch.randint(0, n, (e,), generator=g, device=DEV)
    feat, y = torch.randn(n, dim, c, generator=g, device=DEV), torch.randn(e, dim, generator=g, device=DEV)
    grad = torch.randn(n, table.num_rows, c, generator=g, device=DEV)
    rows, gy = cg_segment_sum(table, feat, y, fidx, None, ptr, n), cg_inner(table, feat, grad, fidx, ptr, node, None, e)

    edges = (2 * some[:, None] + torch.arange(2, device=DEV)).reshape(-1)
    x, big = feat[fidx[edges]].double(), grad[node[edges]].double()
    want, want_gy = torch.zeros(400, table.num_rows, c, dtype=torch.float64, device=DEV), torch.zeros(800, dim, dtype=torch.float64, device=DEV)
    for t in range(table.scale.numel()):
        f = x[:, table.m_feat[t]] * table.scale[t].double()
        want[:, row[t]] += (f * y[edges, table.m_y[t], None].double()).view(400, 2, c).sum(1)
        want_gy[:, table.m_y[t]] += (f * big[:, row[t]]).sum(-1)
    _close(rows[some], want)
    _close(gy[edges], want_gy)


@pytest.mark.parametrize("lmax,c", [(2, 16), (2, 64), (3, 16), (3, 32)])
def test_values_that_are_not_finite_stay_at_their_nodes(lmax, c):
    """Two edges share a warp at 16 channels, and a ring slot outlives its edge: neither may leak into other nodes."""
    dim, table, _, _, path = _tables(lmax, "fwd")
    g = torch.Generator().manual_seed(3)
    n = 301
    ptr = torch.arange(0, 3 * n + 1, 3, dtype=torch.int64, device=DEV)
    feat, y = torch.randn(3 * n, dim, c, generator=g).to(DEV), torch.randn(3 * n, dim, generator=g).to(DEV)
    w, grad = torch.randn(int(path.max()) + 1, c, generator=g).to(DEV), torch.randn(n, dim, c, generator=g).to(DEV)
    fidx = torch.arange(3 * n, device=DEV)
    feat[7], feat[450] = float("inf"), float("nan")
    bad = torch.zeros(n, dtype=torch.bool, device=DEV)
    bad[7 // 3] = bad[450 // 3] = True
    for out in (cg_segment_sum(table, feat, y, fidx, None, ptr, n), cg_segment_mix(table, feat, y, fidx, None, ptr, n, w)[0]):
        assert torch.isfinite(out[~bad]).all() and not torch.isfinite(out[bad]).all(dim=(1, 2)).any()
    gy = cg_inner_mix(table, feat, grad, w, fidx, ptr, None, 3 * n)
    finite = torch.isfinite(gy).all(dim=1)
    assert not finite[7] and not finite[450] and int(finite.sum()) == 3 * n - 2


def test_weight_gradient_of_many_nodes():
    """A warp adds up rows in chains of sixteen nodes, whose sums are added up in 64 bits: at most 112 multiply-adds of random sign
    at l_max 3, each rounded by at most half a unit of the partial sum, which is 2^-24 sqrt(112 / 6) of the result.  In one chain
    over all its nodes, 90 here, the error was 3.6e-7."""
    dim, table, row, comp, path = _tables(3, "fwd")
    g, n, c = torch.Generator(device=DEV).manual_seed(1), 20_000, 128
    e = 3 * n
    ptr, node = torch.arange(0, e + 1, 3, device=DEV), torch.arange(n, device=DEV).repeat_interleave(3)
    fidx = torch.randint(0, n, (e,), generator=g, device=DEV)
    feat, x = (torch.randn(n, dim, c, generator=g, device=DEV) for _ in range(2))
    y, w = torch.randn(e, dim, generator=g, device=DEV), torch.randn(int(path.max()) + 1, c, generator=g, device=DEV)
    want = torch.zeros(w.shape, dtype=torch.float64, device=DEV)
    for t in range(table.scale.numel()):
        term = feat[fidx, table.m_feat[t]].double() * (y[:, table.m_y[t], None].double() * table.scale[t].double())
        want[path[row[t]]] += (x[:, comp[row[t]]].double()[node] * term).sum(0)
    _, got = cg_segment_mix(table, feat, y, fidx, None, ptr, n, w, x)
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -24 * (112 / 6) ** 0.5


def test_keys_without_kernels():
    dim, table, _, _, _ = _tables(2, "fwd")
    assert mix_scratch(table, 10, 64) > 0 and mix_scratch(table, 10, 24) == -1
    odd = Irreps("0e+1e+1o+2e")
    fwd = tp_infos(odd, Irreps("0e+1o+2e"), odd)[0]
    assert mix_scratch(TpTable(fwd.info_Mij_fwd, True, odd.dim, 9, DEV, fwd.info_M_fwd), 10, 64) == -1


def test_tables_that_contradict_their_key_take_the_table_driven_kernels():
    dim, table, _, _, _ = _tables(1, "fwd")
    n, c = 50, 32
    g = torch.Generator().manual_seed(2)
    feat, y, grad = (torch.randn(*s, generator=g).to(DEV) for s in ((n, dim, c), (n, dim), (n, table.num_rows, c)))
    fidx, ptr = torch.arange(n, device=DEV), torch.arange(n + 1, device=DEV)

    def run():
        return cg_segment_sum(table, feat, y, fidx, None, ptr, n), cg_inner(table, feat, grad, fidx, ptr, fidx, None, n)
    want = run()
    table.struct.structure_key = _tables(2, "fwd")[1].key
    for got, expect in zip(run(), want):
        _close(got, expect.double())
