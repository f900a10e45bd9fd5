"""Channel-wise products and their batch-summed form on four channels per thread against the float64 oracle where a block ends:
one row and many, rows without entries and with more than a stage holds, one group of channels and one more than a block has
lanes, sample counts that are no multiple of four or smaller than a block takes, operands off the 16-byte grid."""
import pytest
import torch

from equitorch_b200.ops import batched_sparse_dense_op as gops
from oracle import sparse_ops as oops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _table(g, num_out, entries, rows):
    owner = torch.sort(torch.randint(0, num_out, (entries,), generator=g)).values
    seg = torch.zeros(num_out + 1, dtype=torch.long)
    seg[1:] = torch.cumsum(torch.bincount(owner, minlength=num_out), 0)
    i1, i2 = (torch.randint(0, rows, (entries,), generator=g) for _ in range(2))
    return torch.randn(entries, generator=g), i1, i2, seg


@pytest.mark.parametrize("accumulated", [False, True])
@pytest.mark.parametrize("num_out,entries", [(1, 1), (2, 150), (512, 1024), (512, 1025), (513, 600), (9, 40)])
@pytest.mark.parametrize("n,c", [(1, 4), (3, 132), (70, 64), (257, 128), (40, 12)])
def test_products_against_the_oracle(n, c, num_out, entries, accumulated):
    g = torch.Generator().manual_seed(n * c + entries)
    sc, i1, i2, seg = _table(g, num_out, entries, 7)
    x, y = torch.randn(n, 7, c, generator=g), torch.randn(n, 7, c, generator=g)
    shared = torch.randn(7, c, generator=g)
    scalar = torch.randn(n, 7, generator=g)
    dev = lambda t: t.to(DEV)
    kw = dict(out_accumulated=accumulated)
    for name, second in (("indexed_mul_scale_gather", y), ("indexed_mul_scale_gather", shared), ("indexed_vecsca_scale_gather", scalar)):
        want = getattr(oops, name)(x.double(), second.double(), sc.double(), i1, i2, seg, **kw)
        got = getattr(gops, name)(*map(dev, (x, second, sc, i1, i2, seg)), **kw)
        # float32 sums of up to n * entries / num_out products of unit normals, rounded at their own size: the error relative to
        # the largest sum grows like the root of the number of terms in a chain
        assert got.shape == want.shape
        assert float((got.cpu().double() - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))


def test_operands_off_the_16_byte_grid():
    g = torch.Generator().manual_seed(1)
    sc, i1, i2, seg = (t.to(DEV) for t in _table(g, 5, 20, 7))
    x, y = torch.randn(30 * 7 * 8 + 1, generator=g).to(DEV), torch.randn(30, 7, 8, generator=g).to(DEV)
    off = x[1:].view(30, 7, 8)
    for kw in (dict(), dict(out_accumulated=True)):
        a = gops.indexed_mul_scale_gather(off, y, sc, i1, i2, seg, **kw)
        b = gops.indexed_mul_scale_gather(off.clone(), y, sc, i1, i2, seg, **kw)
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("n,c,num_out", [(1, 4, 1), (511, 4, 1), (513, 4, 1), (70001, 4, 1), (1025, 20, 3), (300, 8, 63), (300, 8, 64), (300, 8, 65), (77, 24, 21)])
def test_rows_that_do_not_fill_a_block(n, c, num_out):
    """One item a sample up to as many as a block has threads and one more; samples that end within a block's step."""
    g = torch.Generator().manual_seed(n + c)
    sc, i1, i2, seg = _table(g, num_out, 2 * num_out + 1, 7)
    x, y, scalar = torch.randn(n, 7, c, generator=g), torch.randn(n, 7, c, generator=g), torch.randn(n, 7, generator=g)
    dev = lambda t: t.to(DEV)
    for name, second in (("indexed_mul_scale_gather", y), ("indexed_vecsca_scale_gather", scalar)):
        want = getattr(oops, name)(x.double(), second.double(), sc.double(), i1, i2, seg)
        got = getattr(gops, name)(*map(dev, (x, second, sc, i1, i2, seg)))
        assert got.shape == want.shape and float((got.cpu().double() - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))
