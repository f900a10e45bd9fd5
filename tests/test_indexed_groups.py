"""Grouping of output rows (vecmat) and of second-operand rows (accumulated outer product) that read the same input rows: the
plans against the plain sums they stand for, on the CPU, and the kernels on such tables against the float64 oracle."""
import numpy as np
import pytest
import torch

from equitorch_b200.ops import indexed_tc_op as tc
from oracle import sparse_ops as oops


def _table(kind, seed):
    """(index1, index2, seg, rows1, rows2, num_out) with index2 = entry number; ``shared``: classes of 1 to 7 rows that read the
    same rows in any order, among them empty ones and rows that read a row twice; ``own``: no two rows read the same."""
    rng = np.random.default_rng(seed)
    rows1, per_row = 11, []
    if kind == "shared":
        for size in (7, 4, 1, 2, 3):
            reads = rng.choice(rows1, rng.integers(1, 6), replace=False).tolist()
            if size == 3:
                reads.append(reads[0])
            per_row += [rng.permutation(reads).tolist() for _ in range(size)]
        per_row += [[], []]
    else:
        per_row = [[r] for r in range(rows1)]
    order = rng.permutation(len(per_row))
    per_row = [per_row[i] for i in order]
    seg = np.concatenate([[0], np.cumsum([len(r) for r in per_row])])
    i1 = torch.tensor([v for r in per_row for v in r])
    return i1, torch.arange(len(i1)), torch.from_numpy(seg), rows1, len(i1), len(per_row)


@pytest.mark.parametrize("cin,cout", [(32, 32), (64, 64), (32, 96), (32, 16), (96, 48)])
@pytest.mark.parametrize("kind", ["shared", "own"])
def test_vecmat_plan_covers_every_entry_once(kind, cin, cout):
    i1, _, seg, rows1, _, num_out = _table(kind, cin + cout)
    plan = tc.VecmatPlan(i1, seg, len(i1), num_out, cin, cout, "cpu")
    chunks, group = cin // 32, plan.group
    assert group * cout <= 128 and (group == 1 or cout % 32 == 0)
    assert group == 1 if kind == "own" or cout % 32 else group > 1 or cout > 64
    rows = plan.group_rows.numpy().reshape(plan.num_groups, group)
    entry = plan.slot_entry.numpy().reshape(-1, group)
    begin, col = plan.kb_begin.numpy(), plan.a_col.numpy()
    assert sorted(rows[rows >= 0].tolist()) == list(range(num_out))
    seen = []
    for g in range(plan.num_groups):
        assert (begin[g + 1] - begin[g]) % chunks == 0
        for slot in range(begin[g] // chunks, begin[g + 1] // chunks):
            read = col[slot * chunks] // cin
            assert col[slot * chunks:(slot + 1) * chunks].tolist() == [read * cin + 32 * q for q in range(chunks)]
            for q in range(group):
                t = entry[slot, q]
                assert (t < 0) == (rows[g, q] < 0)
                if t >= 0:
                    assert int(i1[t]) == read and seg[rows[g, q]] <= t < seg[rows[g, q] + 1]
                    seen.append(int(t))
    assert sorted(seen) == list(range(len(i1)))


@pytest.mark.parametrize("c1,c2", [(32, 32), (64, 32), (96, 64), (32, 128), (64, 128), (256, 64)])
@pytest.mark.parametrize("kind", ["shared", "own"])
def test_outer_plan_covers_every_entry_once(kind, c1, c2):
    # the second operand's rows are the table's output rows, so that classes of them meet the same first-operand rows
    i1, _, seg, rows1, _, num_out = _table(kind, c1 + c2)
    i2 = torch.repeat_interleave(torch.arange(num_out), seg.diff())
    w_seg = torch.arange(len(i1) + 1)
    plan = tc.OuterPlan(None, i1, i2, w_seg, len(i1), len(i1), c1, c2, "cpu")
    first, second, cf, cs = (i2, i1, c2, c1) if plan.swapped else (i1, i2, c1, c2)
    chunks, group = cf // 32, plan.group
    a, b = plan.a_cols.numpy().reshape(-1, 4), plan.b_cols.numpy().reshape(-1, group)
    assert len(a) == len(b) == plan.m_tiles and group * cs <= 128
    ptr, slot = plan.red_ptr.numpy(), plan.red_slot.numpy()
    for w in range(len(i1)):
        for ch in range(chunks):
            units = slot[ptr[w * chunks + ch]:ptr[w * chunks + ch + 1]]
            assert len(units) == 1
            which, at = units[0] >> 24, units[0] & 0xffffff
            assert a[at // 4, at % 4] == int(first[w]) * cf + 32 * ch and b[at // 4, which] == int(second[w]) * cs


@pytest.mark.gpu
@pytest.mark.parametrize("n", [512, 700])
@pytest.mark.parametrize("cin,cout", [(32, 32), (64, 64), (160, 32), (32, 96), (64, 128), (128, 32), (32, 16)])
@pytest.mark.parametrize("kind", ["shared", "own"])
def test_kernels_on_grouped_tables(kind, cin, cout, n):
    from equitorch_b200.ops import batched_sparse_dense_op as gops
    from equitorch_b200.ops.fused_tp_op import check_status
    i1, i2, seg, rows1, rows2, num_out = _table(kind, cin + cout)
    g = torch.Generator().manual_seed(n + cin)
    x, w, sc = torch.randn(n, rows1, cin, generator=g), torch.randn(rows2, cin, cout, generator=g), torch.randn(len(i1), generator=g)
    dev = lambda t: t.to("cuda:0")
    want = oops.indexed_vecmat_scale_gather(x.double(), w.double(), sc.double(), i1, i2, seg)
    got = gops.indexed_vecmat_scale_gather(*map(dev, (x, w, sc, i1, i2, seg)))
    check_status()
    assert float((got.cpu().double() - want).abs().max() / want.abs().max()) < 1e-5
    if cout % 32 == 0:
        y = torch.randn(n, num_out, cout, generator=g)
        back, w_seg = torch.repeat_interleave(torch.arange(num_out), seg.diff()), torch.arange(len(i1) + 1)
        want = oops.indexed_outer_scale_gather(x.double(), y.double(), sc.double(), i1, back, w_seg, out_accumulated=True)
        got = gops.indexed_outer_scale_gather(*map(dev, (x, y, sc, i1, back, w_seg)), out_accumulated=True)
        check_status()
        assert float((got.cpu().double() - want).abs().max() / want.abs().max()) < 1e-5
