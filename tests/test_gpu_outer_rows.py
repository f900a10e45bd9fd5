"""Per-sample outer products at the edges of the row kernel: column counts of 4 to 128 in powers of two (one warp per
output row), row counts that are no multiple of the rows a warp serves at a time, shared operands, an output-row table,
rows without entries - and a column count beside it (12) that stays on the element-wise kernel."""
import pytest
import torch

from equitorch_b200.ops import batched_sparse_dense_op as gops
from oracle import sparse_ops as oops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# a row sums at most 6 products: (6 + 2) roundings of half an ulp of the largest term; bfloat16 rounds the result once
BOUND = {torch.float32: 8 * 2.0 ** -24 * 6, torch.float64: 8 * 2.0 ** -53 * 6, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("n,c1,c2", [(1, 1, 4), (3, 9, 8), (37, 32, 32), (5, 33, 16), (2, 7, 128), (300, 17, 64), (4, 6, 12)])
def test_outer_rows(n, c1, c2, dtype):
    g = torch.Generator().manual_seed(n + c1 + c2)
    seg = torch.tensor([0, 2, 2, 8, 9])
    i1, i2 = torch.randint(0, 3, (9,), generator=g), torch.randint(0, 5, (9,), generator=g)
    sc = torch.randn(9, generator=g, dtype=torch.float64)
    arith = torch.float64 if dtype == torch.float64 else torch.float32
    a, b = torch.randn(n, 3, c1, generator=g).to(dtype), torch.randn(n, 5, c2, generator=g).to(dtype)
    out_rows = torch.tensor([4, 0, 1, 3])
    for x, y, index_out in [(a, b, None), (a, b, out_rows), (a[0], b, None), (a, b[0], None)]:
        size = 4 if index_out is None else 6
        want = oops.indexed_outer_scale_gather(x.double(), y.double(), sc.to(arith).double(), i1, i2, seg, index_out=index_out, out_size=size)
        got = gops.indexed_outer_scale_gather(x.to(DEV), y.to(DEV), sc.to(arith).to(DEV), i1.to(DEV), i2.to(DEV), seg.to(DEV),
                                              index_out=None if index_out is None else index_out.to(DEV), out_size=size)
        assert got.dtype == dtype and got.shape == want.shape
        assert float((got.double().cpu() - want).abs().max()) <= BOUND[dtype] * float(want.abs().max())
